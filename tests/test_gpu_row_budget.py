"""Differentiable steps whose rays hold more rows than the buffers.

A step keeps whole rays in one sub-iteration where its row buffer holds them;
a warp whose window finds no room marches it in the next sub-iteration, and the
second pass marches again.  Such steps, by lanes and by a lane a ray, plain and
cached, against a set compaction batch, whose windows always fit: the same
samples in the same order per ray, so the predictions are equal bit for bit and
the gradients are the same float32 sums in another order.
"""
import numpy as np
import pytest

import frustumvolumecaching_gb300 as fvc
from frustumvolumecaching_gb300.camera import rotation_path
from tests.helpers import small_camera, tiny_model

pytestmark = pytest.mark.gpu


def _step(r, info, pix, tgt, net, n):
    torch = pytest.importorskip("torch")
    g = fvc.Gradients(net)
    pred = torch.zeros((n, 4), dtype=torch.float32, device="cuda")
    loss = r.render_backward(info, pix, tgt, g, pred=pred)
    st = r._render_stats
    assert st.guard_flags == 0
    return loss, pred.cpu().numpy(), [np.asarray(x, np.float64).ravel() for x in g.read()], st


def _compare(one, two):
    (la, pa, ga, sa), (lb, pb, gb, sb) = one, two
    np.testing.assert_array_equal(pa.view(np.uint32), pb.view(np.uint32))
    assert sa.n_samples == sb.n_samples
    assert abs(la - lb) <= 1e-9 * abs(lb)  # float32 terms added in float64
    # float32 sums of n_samples terms in another order: about sqrt(n) 2^-24 of their terms' norm
    for a, b in zip(ga, gb):
        assert np.linalg.norm(a - b) <= 2.0 * np.sqrt(sb.n_samples) * 2.0 ** -24 * np.linalg.norm(b)


# all pixels of the view or 98305 of them; finer steps for more rows a ray; the buffer's rows a ray
CASES = [(320, 300, 96000, 4.0, 160), (700, 601, 98305, 4.0, 137), (1024, 1024, 1 << 20, 2.0, 64), (2048, 1024, 1 << 21, 1.0, 32)]


@pytest.mark.parametrize("W,H,n,finer,rows_a_ray", CASES)
def test_plain_step(W, H, n, finer, rows_a_ray):
    torch = pytest.importorskip("torch")
    loader = fvc.load_data(tiny_model(7, 1))
    steps = fvc.change_sampling_rate(loader.stepsize_info, finer, loader.scene_info)
    rng = np.random.default_rng(5)
    pix = torch.from_numpy(rng.permutation(W * H)[:n].astype(np.int32)).cuda()
    tgt = torch.from_numpy(rng.uniform(0, 1, (n, 3)).astype(np.float32)).cuda()
    info = fvc.raymarch_info(small_camera(1001, W, H, radius=2.5), steps)
    out = []
    for general in (False, True):
        r = fvc.PerformanceRenderer(loader.scene_info, loader.occupancy_grid_morton_bitfield, loader.nerf_network)
        if general:
            r.set_tiling(128, 1 << 24)
            r.set_empty_space_skipping(True)
        out.append(_step(r, info, pix, tgt, loader.nerf_network, n))
    assert out[0][3].n_samples > rows_a_ray * n and out[0][3].n_rounds > 1
    _compare(*out)


@pytest.mark.parametrize("W,H", [(320, 300), (400, 300)])
def test_cached_step(W, H):
    torch = pytest.importorskip("torch")
    loader = fvc.load_data(tiny_model(7, 1))
    steps = fvc.change_sampling_rate(loader.stepsize_info, 4.0, loader.scene_info)
    path = rotation_path(1001, n_frames=2, width=W, height=H)  # the second frame half a degree on: rows of both kinds
    n = W * H
    rng = np.random.default_rng(6)
    pix = torch.from_numpy(rng.permutation(n).astype(np.int32)).cuda()
    tgt = torch.from_numpy(rng.uniform(0, 1, (n, 3)).astype(np.float32)).cuda()
    out = []
    for general in (False, True):
        c0, c1 = fvc.Cache(), fvc.Cache()
        r = fvc.CachePerformanceRenderer(loader.scene_info, loader.occupancy_grid_morton_bitfield, loader.nerf_network, c0, c1)
        r.resizeCache((W, H), steps)
        r.setCacheSettings(fvc.default_cache_settings())
        if general:
            r.set_tiling(128, 1 << 24)
            r.set_empty_space_skipping(True)
        r.initCacheBlockwise(fvc.raymarch_info(path[0], steps))
        r.swapCache()
        out.append(_step(r, fvc.raymarch_info(path[1], steps), pix, tgt, loader.nerf_network, n))
    assert out[0][3].n_samples > 160 * n and out[0][3].n_rounds > 1
    assert out[0][3].n_cache_hits > 0
    _compare(*out)
