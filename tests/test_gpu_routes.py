"""The routes that a call's size picks, against the general one.

A frame of few rays marches several windows a sub-iteration, by 8 lanes a ray
(up to 98304 rays), and composites in blocks (up to 32768); a set compaction
batch keeps one window, empty-space skipping keeps a lane a ray, and the
64-row tiles are another network kernel.  A differentiable step holds whole
rays in one sub-iteration, or marches again with a set batch; its pixel list is
ordered by image tiles (16384 of them at most).  A build searches eight bricks
at once below 1024 tiles and takes the tcgen05 network from 2^18 rays.  The
same arithmetic in the same order per ray: outputs are equal bit for bit, but
for the atomic sums of the gradients.
"""
import threading
from dataclasses import replace

import numpy as np
import pytest

import frustumvolumecaching_gb300 as fvc
from frustumvolumecaching_gb300 import model as fmodel
from oracle import oracle as orc
from tests.helpers import small_camera, tiny_model

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def models(tmp_path_factory):
    """A fog, three cascades, and a scene whose rays end by opacity."""
    sm = fmodel.SyntheticModel(replace(fmodel.spec_tiny(seed=7, nlvl=1), name="opaque"))
    sm.build_occupancy()
    sm.base[1][0] = (sm.base[1][0].astype(np.float32) * 1350).astype(np.float16)  # log-densities of about 4.5
    opaque = sm.write(str(tmp_path_factory.mktemp("routes") / "opaque"))
    return {"fog": fvc.load_data(tiny_model(7, 1)), "cascades": fvc.load_data(tiny_model(9, 3)), "opaque": fvc.load_data(opaque)}


def _general(r):
    r.set_tiling(64, 1 << 24)
    r.set_empty_space_skipping(True)


def _frame(r, cam, loader):
    buf = fvc.RenderBuffer(cam["resolution"])
    r.render(fvc.raymarch_info(cam, loader.stepsize_info), buf)
    assert r._render_stats.guard_flags == 0
    return buf, r._render_stats.n_samples


def _same(a, b):
    np.testing.assert_array_equal(a[0].ray_counts, b[0].ray_counts)
    np.testing.assert_array_equal(a[0].results.view(np.uint32), b[0].results.view(np.uint32))
    np.testing.assert_array_equal(a[0].image, b[0].image)
    assert a[1] == b[1]


# around a march block, the compositing's line (32768 rays) and the march's (98304), and a frame of few windows
SIZES = [(1, 1), (33, 1), (37, 21), (181, 181), (182, 181), (313, 314), (314, 314), (811, 405)]


@pytest.mark.parametrize("W,H", SIZES)
@pytest.mark.parametrize("scene", ["fog", "cascades", "opaque"])
def test_plain_frame(models, scene, W, H):
    loader = models[scene]
    cam = small_camera(1601, W, H)
    out = []
    for general in (False, True):
        r = fvc.PerformanceRenderer(loader.scene_info, loader.occupancy_grid_morton_bitfield, loader.nerf_network)
        if general:
            _general(r)
        out.append(_frame(r, cam, loader))
    _same(*out)


@pytest.mark.parametrize("W,H", SIZES[2:])
@pytest.mark.parametrize("scene", ["cascades", "opaque"])
def test_cached_frame(models, scene, W, H):
    loader = models[scene]
    out = []
    for general in (False, True):
        c0, c1 = fvc.Cache(), fvc.Cache()
        r = fvc.CachePerformanceRenderer(loader.scene_info, loader.occupancy_grid_morton_bitfield, loader.nerf_network, c0, c1)
        r.resizeCache((W, H), loader.stepsize_info)
        r.resizeRenderbuffers((W, H))
        r.setCacheSettings(fvc.default_cache_settings())
        if general:
            r.set_tiling(128, 1 << 24)
            r.set_empty_space_skipping(True)
        r.initCache(fvc.raymarch_info(small_camera(1001, W, H), loader.stepsize_info))  # the per-ray fill takes the march's route too
        fill = [x.copy() for x in c1.read()]
        n = r._init_stats.n_bricks_set
        r.swapCache()
        out.append((_frame(r, small_camera(1002, W, H), loader), fill, n))
    _same(out[0][0], out[1][0])
    assert out[0][2] == out[1][2]
    for k in (0, 1):
        np.testing.assert_array_equal(out[0][1][k].view(np.uint32), out[1][1][k].view(np.uint32))
    n = out[0][2]
    np.testing.assert_array_equal(out[0][1][2][:n].view(np.uint8), out[1][1][2][:n].view(np.uint8))


@pytest.mark.parametrize("W,H", [(5, 3), (61, 43), (250, 167)])
def test_bf16_frame(models, W, H):
    """The rows that share a network tile differ between the two."""
    loader = models["fog"]
    cam = small_camera(1601, W, H)
    out = []
    for batch in (0, 1024):
        r = fvc.PerformanceRenderer(loader.scene_info, loader.occupancy_grid_morton_bitfield, loader.nerf_network)
        r.set_precision(fvc.PerformanceRenderer.BF16)
        r.set_tiling(128, batch)
        out.append(_frame(r, cam, loader))
    _same(*out)


@pytest.mark.parametrize("W,H,n", [(8, 8, 1), (40, 24, 33), (64, 64, 4096), (2051, 517, 4099), (700, 601, 98305)])
@pytest.mark.parametrize("precision", [0, 1], ids=["fp16", "bf16"])
def test_differentiable_step(models, W, H, n, precision):
    """2051x517 pixels have more than 16384 tiles of 8x8.  Gradients: float32
    atomic sums of m terms in another order differ by about sqrt(m) 2^-24 of
    their terms' norm, 6e-5 at m = 2^20."""
    torch = pytest.importorskip("torch")
    loader = models["fog"]
    rng = np.random.default_rng(3)
    pix = torch.from_numpy(rng.choice(W * H, n, replace=False).astype(np.int32)).cuda()
    tgt = torch.from_numpy(rng.uniform(0, 1, (n, 3)).astype(np.float32)).cuda()
    info = fvc.raymarch_info(small_camera(1001, W, H), loader.stepsize_info)
    out = []
    for general in (False, True):
        r = fvc.PerformanceRenderer(loader.scene_info, loader.occupancy_grid_morton_bitfield, loader.nerf_network)
        r.set_precision(precision)
        if general:
            r.set_tiling(128, 1 << 24)
            r.set_empty_space_skipping(True)
        g = fvc.Gradients(loader.nerf_network)
        pred = torch.zeros((n, 4), dtype=torch.float32, device="cuda")
        loss = r.render_backward(info, pix, tgt, g, pred=pred)
        out.append((loss, pred.cpu().numpy(), [np.asarray(x, np.float64).ravel() for x in g.read()]))
    (la, pa, ga), (lb, pb, gb) = out
    np.testing.assert_array_equal(pa.view(np.uint32), pb.view(np.uint32))
    assert abs(la - lb) <= 1e-5 * abs(lb)
    for a, b in zip(ga, gb):
        assert np.linalg.norm(a - b) <= 1e-4 * np.linalg.norm(b)


@pytest.mark.parametrize("W,H", [(260, 250), (520, 514)])
def test_build_networks_and_search_agree(models, W, H):
    """1056 tiles at the start (the one-brick search first, the eight-brick one
    as tiles end) against the oracle; 4290 tiles are past 2^18 rays, where the
    build picks tcgen05."""
    loader = models["opaque" if W > 512 else "fog"]
    cam = small_camera(1001, W, H)
    out = []
    for path in (None, False, True):
        c0, c1 = fvc.Cache(), fvc.Cache()
        r = fvc.CachePerformanceRenderer(loader.scene_info, loader.occupancy_grid_morton_bitfield, loader.nerf_network, c0, c1)
        r.resizeCache((W, H), loader.stepsize_info)
        if path is not None:
            r.set_build_network_path(path)
        r.initCacheBlockwise(fvc.raymarch_info(cam, loader.stepsize_info))
        out.append(([x.copy() for x in c1.read()], r._init_stats.n_bricks_set))
    for x, n in out[1:]:
        assert n == out[0][1]
        np.testing.assert_array_equal(x[0], out[0][0][0])
        np.testing.assert_array_equal(x[1].view(np.uint32), out[0][0][1].view(np.uint32))
        np.testing.assert_array_equal(x[2][:n].view(np.uint8), out[0][0][2][:n].view(np.uint8))
    if W < 512:
        oc = orc.OracleModel(tiny_model(7, 1)).cache_build(cam)
        np.testing.assert_array_equal(out[0][0][0].ravel(), oc.packed_index)
        np.testing.assert_array_equal(out[0][0][1].ravel().view(np.uint32), oc.known_ranges.view(np.uint32))


def test_queries_share_the_scratch(models):
    """Queries of growing and shrinking sizes, past the kept scratch (2^24
    floats), and from four threads at once, against one at a time."""
    net = models["fog"].nerf_network
    rng = np.random.default_rng(9)
    pos = rng.uniform(0, 1, (1_700_000, 3)).astype(np.float32)
    d01 = rng.uniform(0, 1, pos.shape).astype(np.float32)
    whole = net.inference(pos, d01)
    sizes = [1, 4097, 33, 100_000, 2]
    for n in sizes:
        np.testing.assert_array_equal(net.inference(pos[:n], d01[:n]), whole[:n])
    np.testing.assert_array_equal(net.density(pos[:1000]), whole[:1000, 3])
    got = {}

    def query(t):
        got[t] = [net.inference(pos[t:t + n], d01[t:t + n]) for n in sizes * 4]

    threads = [threading.Thread(target=query, args=(t,)) for t in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for t in range(4):
        for n, x in zip(sizes * 4, got[t]):
            np.testing.assert_array_equal(x, whole[t:t + n])
