"""Statistics and the sample guard do not depend on how many march windows a
sub-iteration holds: rows and steps are counted up to the window a ray ended
in, whether the rays behind it were marched further or not.  Frames, fills,
batches and differentiable steps of an opaque scene and of a fog against a set
compaction batch, which marches one window at a time."""
from dataclasses import replace

import numpy as np
import pytest

import frustumvolumecaching_gb300 as fvc
from frustumvolumecaching_gb300 import model as fmodel
from frustumvolumecaching_gb300.camera import rotation_path
from tests.helpers import small_camera, tiny_model

pytestmark = pytest.mark.gpu

FIELDS = ("n_samples", "n_resamples", "n_cache_hits", "n_dropped", "n_steps", "guard_flags", "n_miss_outside_fov", "n_miss_outside_depth",
          "n_miss_before_near", "n_miss_beyond_known", "n_drop_brick_unset", "n_drop_voxel_empty", "n_drop_alpha")
SIZES = [(33, 1), (37, 21), (182, 181), (320, 313)]


@pytest.fixture(scope="module")
def models(tmp_path_factory):
    sm = fmodel.SyntheticModel(replace(fmodel.spec_tiny(seed=7, nlvl=1), name="opaque"))
    sm.build_occupancy()
    sm.base[1][0] = (sm.base[1][0].astype(np.float32) * 1350).astype(np.float16)  # log-densities of about 4.5
    opaque = sm.write(str(tmp_path_factory.mktemp("statistics") / "opaque"))
    return {"fog": fvc.load_data(tiny_model(7, 1)), "opaque": fvc.load_data(opaque)}


def _stats(r):
    s = r._render_stats
    return {f: int(getattr(s, f)) for f in FIELDS}


def _renderer(loader, general, kind=fvc.PerformanceRenderer, *caches):
    r = kind(loader.scene_info, loader.occupancy_grid_morton_bitfield, loader.nerf_network, *caches)
    if general:
        r.set_tiling(128, 1 << 24)
    return r


def _render(r, loader, cam):
    r.render(fvc.raymarch_info(cam, loader.stepsize_info), fvc.RenderBuffer(cam["resolution"]))
    return _stats(r)


@pytest.mark.parametrize("W,H", SIZES)
@pytest.mark.parametrize("scene", ["fog", "opaque"])
def test_plain_frame(models, scene, W, H):
    loader, cam = models[scene], small_camera(1601, W, H)
    one, two = (_render(_renderer(loader, general), loader, cam) for general in (False, True))
    assert one == two and one["n_resamples"] >= one["n_samples"] > 0


@pytest.mark.parametrize("W,H", SIZES[1:])
@pytest.mark.parametrize("kind,fused", [(fvc.CachePerformanceRenderer, True), (fvc.CachePerformanceRenderer, False), (fvc.CacheBasicRenderer, True)],
                         ids=["fused", "classify", "basic"])
def test_cached_frame_and_fill(models, kind, fused, W, H):
    loader = models["opaque"]
    path = rotation_path(1001, n_frames=2, width=W, height=H)
    out = []
    for general in (False, True):
        c0, c1 = fvc.Cache(), fvc.Cache()
        r = _renderer(loader, general, kind, c0, c1)
        r.set_fused_classify(fused)
        r.resizeCache((W, H), loader.stepsize_info)
        r.resizeRenderbuffers((W, H))
        r.setCacheSettings(fvc.default_cache_settings())
        r.initCache(fvc.raymarch_info(path[0], loader.stepsize_info))
        fill = _stats(r)
        r.swapCache()
        out.append((fill, _render(r, loader, path[1])))
    assert out[0] == out[1]
    assert out[0][0]["n_steps"] > 0 and out[0][1]["n_cache_hits"] > 0 and out[0][1]["n_resamples"] > 0


def test_batch(models):
    torch = pytest.importorskip("torch")
    loader = models["opaque"]
    infos = [fvc.raymarch_info(small_camera(1601 + v, 60 - 7 * v, 40), loader.stepsize_info) for v in range(3)]
    n = sum((60 - 7 * v) * 40 for v in range(3))
    out = []
    for general in (False, True):
        r = _renderer(loader, general)
        r.render_batch(infos, results=torch.zeros((n, 4), dtype=torch.float32, device="cuda"))
        r.synchronize()
        out.append(_stats(r))
    assert out[0] == out[1] and out[0]["n_samples"] > 0


@pytest.mark.parametrize("W,H", SIZES[1:])
def test_differentiable_step(models, W, H):
    """One sub-iteration, or as many as windows: both passes' rows and steps."""
    torch = pytest.importorskip("torch")
    loader = models["opaque"]
    pix = torch.arange(W * H, dtype=torch.int32, device="cuda")
    tgt = torch.zeros((W * H, 3), dtype=torch.float32, device="cuda")
    out = []
    for general in (False, True):
        r = _renderer(loader, general)
        r.render_backward(fvc.raymarch_info(small_camera(1601, W, H), loader.stepsize_info), pix, tgt, fvc.Gradients(loader.nerf_network))
        out.append(_stats(r))
    frame = _render(_renderer(loader, True), loader, small_camera(1601, W, H))
    assert out[0] == out[1] and out[0]["n_samples"] == frame["n_samples"]
    for f in ("n_resamples", "n_steps"):
        assert out[0][f] == 2 * frame[f]


@pytest.mark.parametrize("W,H", [(37, 21), (320, 313)])
@pytest.mark.parametrize("what", ["plain", "cached", "fill"])
def test_sample_guard(models, what, W, H):
    """The smallest limit that does not fire is the same, below the rows of a sub-iteration."""
    loader = models["opaque"]
    path = rotation_path(1001, n_frames=2, width=W, height=H)
    limits = []
    for general in (False, True):
        r = _renderer(loader, general) if what == "plain" else _renderer(loader, general, fvc.CachePerformanceRenderer, fvc.Cache(), fvc.Cache())
        info = fvc.raymarch_info(path[0], loader.stepsize_info)
        if what != "plain":
            r.resizeCache((W, H), loader.stepsize_info)
            r.resizeRenderbuffers((W, H))
            r.setCacheSettings(fvc.default_cache_settings())
            r.initCacheBlockwise(info)
            r.swapCache()
            r.resizeCache((W, H), loader.stepsize_info)

        def fires(limit):
            r.set_max_samples_per_ray(limit)
            if what != "fill":
                return bool(_render(r, loader, path[1])["guard_flags"] & 1)
            try:
                r.initCache(info)
            except fvc._lib.FvcError as e:
                assert "guard" in str(e)
                return True
            return False

        lo, hi = 0, 496  # fires above 0 samples; the rows of a whole sub-iteration do not
        assert not fires(hi)
        while hi - lo > 1:
            mid = (lo + hi) // 2
            lo, hi = (mid, hi) if fires(mid) else (lo, mid)
        limits.append(hi)
    assert limits[0] == limits[1] > 1
