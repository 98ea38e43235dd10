"""Weight gradients of a large differentiable step against its rays in steps of
2048 added up in float64.  The adjoint's tensor cores truncate their sums, some
5e-7 of the value a tile of 128 rows, so a CTA adds them to the float32 blobs
every few tiles; added once a launch they would be 4e-5 off here (some 70 tiles
a CTA)."""
import numpy as np
import pytest

import frustumvolumecaching_gb300 as fvc
from tests.helpers import small_camera, tiny_model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [fvc.PerformanceRenderer.FP16, fvc.PerformanceRenderer.BF16], ids=["fp16", "bf16"])
def test_weight_gradients_of_a_large_step(precision):
    torch = pytest.importorskip("torch")
    loader = fvc.load_data(tiny_model(7, 1))
    W, H, n, part = 256, 256, 32768, 2048
    rng = np.random.default_rng(8)
    pix = torch.from_numpy(rng.permutation(W * H)[:n].astype(np.int32)).cuda()
    tgt = torch.from_numpy(rng.uniform(0, 1, (n, 3)).astype(np.float32)).cuda()
    info = fvc.raymarch_info(small_camera(1001, W, H), loader.stepsize_info)
    r = fvc.PerformanceRenderer(loader.scene_info, loader.occupancy_grid_morton_bitfield, loader.nerf_network)
    r.set_precision(precision)

    def weights(a, b):
        g = fvc.Gradients(loader.nerf_network)
        r.render_backward(info, pix[a:b].contiguous(), tgt[a:b].contiguous(), g)
        return [np.asarray(x, np.float64).ravel() for x in g.read()[1:]]

    whole = weights(0, n)
    parts = [weights(a, a + part) for a in range(0, n, part)]
    for k, name in enumerate(("base", "head")):
        ref = np.mean([p[k] for p in parts], axis=0)  # a step's gradient is its rays' mean
        # two tiles' truncation (1e-6), and at most 2^14 float32 additions to the blobs: sqrt(2^14) 2^-24 = 8e-6
        assert np.linalg.norm(whole[k] - ref) <= 1e-5 * np.linalg.norm(ref), name
