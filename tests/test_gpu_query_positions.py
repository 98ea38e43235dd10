"""Network queries at positions outside [0, 1]^3: the positions are the
caller's, so a NaN, an infinity or a coordinate far outside reads inside its
level of the table.  The other rows are those of a query without them, bit for
bit; a position that is not finite has NaN features, as its fractions are."""
import dataclasses

import numpy as np
import pytest

import frustumvolumecaching_gb300 as fvc
from frustumvolumecaching_gb300 import model as fmodel
from tests.helpers import tiny_model

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=["2_features", "4_features"])
def net(request):
    if request.param == "2_features":
        return fvc.load_data(tiny_model(7, 1)).nerf_network
    s = fmodel.spec_tiny(seed=41, nlvl=1)
    return fvc.load_data(fmodel.ensure_model(dataclasses.replace(s, name=f"{s.name}_f4", n_levels=8, F=4, per_level_scale=2.0))).nerf_network


def test_positions_outside_the_grid(net):
    rng = np.random.default_rng(15)
    pos = rng.uniform(0, 1, (4097, 3)).astype(np.float32)
    d01 = rng.uniform(0, 1, pos.shape).astype(np.float32)
    ref, ref_f = net.inference(pos, d01), net.debug_encode(pos)[0]
    odd = np.array([np.nan, np.inf, -np.inf, 3e38, -3e38, 3e6, -3e6, 900.0, -900.0, 2.5, -1.5, 1.0 + 1e-6, -0.04], np.float32)
    at = rng.permutation(len(pos))[:4 * len(odd)].reshape(len(odd), 4)
    bad = pos.copy()
    for v, rows in zip(odd, at):
        for axis, row in enumerate(rows):  # each axis, then all three
            bad[row, axis if axis < 3 else slice(None)] = v
    out, f = net.inference(bad, d01), net.debug_encode(bad)[0]
    rest = np.setdiff1d(np.arange(len(pos)), at)
    np.testing.assert_array_equal(out[rest], ref[rest])
    np.testing.assert_array_equal(f[rest], ref_f[rest])
    finite = np.isfinite(bad).all(1)
    assert np.isnan(f[~finite]).all()
    near = np.abs(bad).max(1) <= 1000  # scale * x below 2^22 at every level: fractions in [0, 1)
    # a fraction in [0, 1) gives a mean of table entries, which stay below 0.011
    assert np.abs(f[near & finite]).max() < 0.02
    np.testing.assert_array_equal(net.density(bad)[rest], ref[rest, 3])
