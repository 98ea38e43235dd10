"""Allocations that fail: a differentiable step without the memory for its
rays' whole rows takes a frame's rows and marches in more sub-iterations, and a
resize without the memory for every march window takes one window's; both give
the same results.  A step whose other buffers fail, and a resize that fails,
leave the renderer usable at any size.  A per-ray cache fill allocates for its
own rows, not for those a step has left the renderer with."""
import numpy as np
import pytest

import frustumvolumecaching_gb300 as fvc
from frustumvolumecaching_gb300 import _lib as L
from tests.helpers import small_camera, tiny_model

pytestmark = pytest.mark.gpu

FVC_ERR_OOM = 3


@pytest.fixture(scope="module")
def loader():
    return fvc.load_data(tiny_model(7, 1))


def _renderer(loader):
    return fvc.PerformanceRenderer(loader.scene_info, loader.occupancy_grid_morton_bitfield, loader.nerf_network)


class failing:
    """The k-th allocation from here on fails."""

    def __init__(self, k):
        self.k = k

    def __enter__(self):
        assert L.load().fvc_debug_fail_allocation(self.k) == 0

    def __exit__(self, *_):
        L.load().fvc_debug_fail_allocation(-1)


# the step's buffers: ray rows, four of the rows, three of the adjoint's; then the pixel list's three and the rays'
ROW_BUFFERS = range(8)


def test_step_without_the_memory_for_whole_rays(loader):
    torch = pytest.importorskip("torch")
    W, H, n = 1024, 1024, 200_000  # 128 rows a ray are more than a frame of this size has
    rng = np.random.default_rng(8)
    pix = torch.from_numpy(rng.permutation(W * H)[:n].astype(np.int32)).cuda()
    tgt = torch.from_numpy(rng.uniform(0, 1, (n, 3)).astype(np.float32)).cuda()
    info = fvc.raymarch_info(small_camera(1001, W, H), loader.stepsize_info)

    def step(r):
        g = fvc.Gradients(loader.nerf_network)
        pred = torch.zeros((n, 4), dtype=torch.float32, device="cuda")
        loss = r.render_backward(info, pix, tgt, g, pred=pred)
        return loss, pred.cpu().numpy(), [np.asarray(x, np.float64).ravel() for x in g.read()], r._render_stats.n_samples

    def same(a, b):
        np.testing.assert_array_equal(a[1].view(np.uint32), b[1].view(np.uint32))
        assert abs(a[0] - b[0]) <= 1e-9 * abs(b[0])  # float32 terms added in float64
        for x, y in zip(a[2], b[2]):  # float32 sums of n_samples terms in another order
            assert np.linalg.norm(x - y) <= 2.0 * np.sqrt(b[3]) * 2.0 ** -24 * np.linalg.norm(y)

    ref = step(_renderer(loader))
    for k in [*ROW_BUFFERS, 8, 11]:
        r = _renderer(loader)
        r.resizeRenderbuffers((W, H))
        g = fvc.Gradients(loader.nerf_network)
        if k in ROW_BUFFERS:
            pred = torch.zeros((n, 4), dtype=torch.float32, device="cuda")
            with failing(k):
                loss = r.render_backward(info, pix, tgt, g, pred=pred)
            assert r._render_stats.n_rounds > 1
            same((loss, pred.cpu().numpy(), [np.asarray(x, np.float64).ravel() for x in g.read()]), ref)
        else:
            with failing(k), pytest.raises(L.FvcError) as e:
                r.render_backward(info, pix, tgt, g)
            assert e.value.code == FVC_ERR_OOM
        same(step(r), ref)


def test_resize_without_the_memory_for_every_window(loader):
    cam = small_camera(1001, 48, 40)
    info = fvc.raymarch_info(cam, loader.stepsize_info)
    ref = fvc.RenderBuffer((48, 40))
    _renderer(loader).render(info, ref)
    for k in range(5, 10):  # results, image, counts and two states come first
        r, buf = _renderer(loader), fvc.RenderBuffer((48, 40))
        with failing(k):
            r.render(info, buf)
        np.testing.assert_array_equal(buf.results.view(np.uint32), ref.results.view(np.uint32))
        np.testing.assert_array_equal(buf.ray_counts, ref.ray_counts)


def test_failed_resize_then_the_size_before(loader):
    """The renderer has no buffers after a resize that failed, so the size it had is resized to again."""
    small, large = small_camera(1001, 32, 24), small_camera(1001, 48, 40)
    ref = fvc.RenderBuffer((32, 24))
    r = _renderer(loader)
    r.render(fvc.raymarch_info(small, loader.stepsize_info), ref)
    for k in (0, 3, 4, 10):
        with failing(k), pytest.raises(L.FvcError):
            r.render(fvc.raymarch_info(large, loader.stepsize_info), fvc.RenderBuffer((48, 40)))
        buf = fvc.RenderBuffer((32, 24))
        r.render(fvc.raymarch_info(small, loader.stepsize_info), buf)
        np.testing.assert_array_equal(buf.results.view(np.uint32), ref.results.view(np.uint32))


def test_fill_after_a_step_allocates_for_its_own_rows(loader):
    torch = pytest.importorskip("torch")
    W = H = 512
    info = fvc.raymarch_info(small_camera(1001, W, H), loader.stepsize_info)
    r = fvc.CachePerformanceRenderer(loader.scene_info, loader.occupancy_grid_morton_bitfield, loader.nerf_network, fvc.Cache(), fvc.Cache())
    r.setCacheSettings(fvc.default_cache_settings())
    for _ in range(2):
        r.resizeCache((W, H), loader.stepsize_info)
        r.swapCache()
    r.initCacheBlockwise(info)
    r.swapCache()
    pix = torch.arange(W * H, dtype=torch.int32, device="cuda")
    tgt = torch.zeros((W * H, 3), dtype=torch.float32, device="cuda")
    r.render_backward(info, pix, tgt, fvc.Gradients(loader.nerf_network))  # 2^25 rows
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    r.initCache(info)
    # 2^21 rows of 18 bytes (38 MB) and a few bytes a brick; for 2^25 rows it would be 604 MB
    assert free - torch.cuda.mem_get_info()[0] < 150 << 20
    assert r._init_stats.n_bricks_set > 0
