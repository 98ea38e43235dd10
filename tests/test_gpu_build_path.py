"""The cache builds' network path: each choice, and back to the choice by size."""
import numpy as np
import pytest

import frustumvolumecaching_gb300 as fvc
from frustumvolumecaching_gb300 import _lib as L
from tests.helpers import small_camera, tiny_model

pytestmark = pytest.mark.gpu


def test_the_choice_by_size_can_be_taken_again():
    loader = fvc.load_data(tiny_model(7, 1))
    info = fvc.raymarch_info(small_camera(1001, 64, 48), loader.stepsize_info)
    out = fvc.Cache()
    r = fvc.CachePerformanceRenderer(loader.scene_info, loader.occupancy_grid_morton_bitfield, loader.nerf_network, fvc.Cache(), out)
    r.resizeCache((64, 48), loader.stepsize_info)
    builds = []
    for path in (None, True, None, False, None):
        r.set_build_network_path(path)
        r.initCacheBlockwise(info)
        builds.append([x.copy() for x in out.read()[:2]])
    for b in builds[1:]:
        for x, y in zip(b, builds[0]):
            np.testing.assert_array_equal(x, y)
    for path in (-2, 2):
        with pytest.raises(L.FvcError):
            L.check(L.load().fvc_renderer_set_build_network_path(r.handle, path))
