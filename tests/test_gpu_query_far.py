"""Network queries at finite positions far outside [0, 1]^3: their cells and
fractions are those of the float32 products, as the oracle takes them, up to
coordinates that an integer still holds; dense levels wrap by their size."""
import dataclasses

import numpy as np
import pytest

import frustumvolumecaching_gb300 as fvc
from frustumvolumecaching_gb300 import model as fmodel
from oracle import oracle as orc
from tests.helpers import tiny_model

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=["2_features", "4_features"])
def model(request):
    d = tiny_model(7, 1)
    if request.param == "4_features":
        s = fmodel.spec_tiny(seed=41, nlvl=1)
        d = fmodel.ensure_model(dataclasses.replace(s, name=f"{s.name}_f4", n_levels=8, F=4, per_level_scale=2.0))
    return fvc.load_data(d).nerf_network, orc.OracleModel(d)


@pytest.mark.parametrize("reach", [1.0, 1.5, 40.0, 1e3, 3e4])
def test_far_positions(model, reach):
    net, om = model
    rng = np.random.default_rng(int(reach))
    pos = rng.uniform(-reach, reach, (2051, 3)).astype(np.float32)
    pos[::3] = rng.uniform(0, 1, pos[::3].shape)  # inside and outside in one warp
    pos[1::3, 1:] = rng.uniform(0, 1, pos[1::3, 1:].shape)  # one axis outside
    ref = om.hash_encode(pos)[:, :32]
    # fp16 features of table entries below 0.011: half a unit in the last place is 4e-6, float32 sums a tenth of it
    assert np.abs(net.debug_encode(pos)[0] - ref).max() < 3e-5
