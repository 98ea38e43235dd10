"""A hash grid whose finest levels have more than 2^22 cells an axis (16 levels
a factor of 2.5 apart: 6 and 15 million), where a cell and its fraction come
from conversions: network queries, renders on each network path, a cache build
and the adjoint against the oracle, for both grids."""
import dataclasses

import numpy as np
import pytest

import frustumvolumecaching_gb300 as fvc
from frustumvolumecaching_gb300 import model as fmodel
from oracle import oracle as orc
from tests.helpers import small_camera

pytestmark = pytest.mark.gpu

W, H = 48, 40


@pytest.fixture(scope="module", params=["2_features", "4_features"])
def model(request):
    s = fmodel.spec_tiny(seed=43, nlvl=1)
    s = dataclasses.replace(s, name=f"{s.name}_fine", per_level_scale=2.5)
    if request.param == "4_features":
        s = dataclasses.replace(s, name=f"{s.name}_f4", n_levels=8, F=4, per_level_scale=7.0)
    d = fmodel.ensure_model(s)
    assert fmodel.SyntheticModel(s).levels[-1].scale > 1 << 22
    return fvc.load_data(d), orc.OracleModel(d), d


def test_queries(model):
    loader, om, _ = model
    rng = np.random.default_rng(3)
    pos = rng.uniform(0, 1, (4000, 3)).astype(np.float32)
    d01 = rng.uniform(0, 1, (4000, 3)).astype(np.float32)
    assert np.abs(loader.nerf_network.inference(pos, d01) - om.inference(pos, d01)).max() <= 2e-3  # the networks' fp16, as for other grids


@pytest.mark.parametrize("path", ["tc128", "tc64", "mma", "bf16", "fp8"])
def test_plain_frame(model, path):
    loader, om, _ = model
    cam = small_camera(1001, W, H)
    r = fvc.PerformanceRenderer(loader.scene_info, loader.occupancy_grid_morton_bitfield, loader.nerf_network)
    if path == "mma":
        r.set_network_path(False)
    elif path in ("bf16", "fp8"):
        r.set_precision(r.BF16 if path == "bf16" else r.FP8_E4M3)
    else:
        r.set_tiling(int(path[2:]), 0)
    buf = fvc.RenderBuffer((W, H))
    r.render(fvc.raymarch_info(cam, loader.stepsize_info), buf)
    ref, ns, _ = om.render_plain(cam)
    np.testing.assert_array_equal(buf.ray_counts[..., 0], ns)
    assert np.abs(buf.results - ref).max() <= (2e-2 if path == "fp8" else 2e-3)  # the precisions' bounds for other grids


@pytest.mark.parametrize("build_tc", [False, True])
def test_cached_frame(model, build_tc):
    loader, om, _ = model
    cam = small_camera(1001, W, H)
    r = fvc.CachePerformanceRenderer(loader.scene_info, loader.occupancy_grid_morton_bitfield, loader.nerf_network, fvc.Cache(), fvc.Cache())
    r.resizeCache((W, H), loader.stepsize_info)
    r.setCacheSettings(fvc.default_cache_settings())
    r.set_build_network_path(build_tc)
    info = fvc.raymarch_info(cam, loader.stepsize_info)
    r.initCacheBlockwise(info)
    r.swapCache()
    buf = fvc.RenderBuffer((W, H))
    r.render(info, buf)
    ref, counts = om.render_cached(cam, om.cache_build(cam))
    np.testing.assert_array_equal(buf.ray_counts[..., :2], counts[..., :2])
    assert np.abs(buf.results - ref).max() <= 2e-3


@pytest.mark.parametrize("tcgen05", [True, False], ids=["tcgen05", "mma_sync"])
def test_adjoint(model, tcgen05):
    torch = pytest.importorskip("torch")
    loader, _, d = model
    if loader.nerf_network.properties()["n_levels"] != 16:
        pytest.skip("the adjoint is built for 16 levels of 2 features")
    rng = np.random.default_rng(13)
    cam = small_camera(1001, 32, 32)
    pix = rng.choice(32 * 32, 384, replace=False).astype(np.int32)
    tgt = rng.uniform(0, 1, (384, 3)).astype(np.float32)
    r = fvc.PerformanceRenderer(loader.scene_info, loader.occupancy_grid_morton_bitfield, loader.nerf_network)
    r.set_network_path(tcgen05)
    g = fvc.Gradients(loader.nerf_network)
    r.render_backward(fvc.raymarch_info(cam, loader.stepsize_info), torch.from_numpy(pix).cuda(), torch.from_numpy(tgt).cuda(), g)
    _, *ref, _ = orc.OracleModel(d, mimic_fp16=True).loss_grad(cam, pix, tgt)
    for a, b in zip(g.read(), ref):
        assert np.linalg.norm(a.astype(np.float64) - b) < 2e-3 * np.linalg.norm(b)  # as for other grids
