"""The occupancy bitfield is the model's device memory, which a program may
write (LoaderData::occupancy_grid_morton_bitfield, fvc_model_properties): what
is rendered, built or queried afterwards is of the cells as they are then.  A
model whose bits are overwritten by another's equals that one, bit for bit."""
import ctypes as C
from dataclasses import replace

import numpy as np
import pytest

import frustumvolumecaching_gb300 as fvc
from frustumvolumecaching_gb300 import _lib as L
from frustumvolumecaching_gb300 import model as fmodel
from frustumvolumecaching_gb300.camera import rotation_path
from tests.helpers import small_camera

pytestmark = pytest.mark.gpu

W, H = 61, 43


def _bits(loader):
    torch = pytest.importorskip("torch")
    p = loader.nerf_network.properties()

    class View:
        __cuda_array_interface__ = {"data": (p["occupancy_bitfield"], False), "shape": (p["occupancy_bytes"],), "typestr": "|u1", "version": 3}

    return torch.as_tensor(View(), device="cuda")


@pytest.fixture(params=[1, 3], ids=["one_cascade", "three_cascades"])
def pair(request, tmp_path):
    """The same networks with two occupancies, in blocks of 4^3 cells and single cells."""
    out = []
    for k in (0, 1):
        sm = fmodel.SyntheticModel(replace(fmodel.spec_tiny(seed=7, nlvl=request.param), name=f"occupancy{k}"))
        rng = np.random.default_rng([7, k])
        occ = rng.random((request.param, 32, 32, 32)) < 0.2
        for axis in (1, 2, 3):
            occ = occ.repeat(4, axis)
        occ ^= rng.random(occ.shape) < 0.01
        sm.occupancy = occ.reshape(request.param, -1).astype(np.uint8)
        out.append(fvc.load_data(sm.write(str(tmp_path / str(k)))))
    return out


def _everything(loader, torch):
    """A frame, a batch, a frame without allocations, a step, both cache builds and a cached frame."""
    steps, out = loader.stepsize_info, []
    path = rotation_path(1001, n_frames=2, width=W, height=H)
    infos = [fvc.raymarch_info(c, steps) for c in path]
    r = fvc.PerformanceRenderer(loader.scene_info, loader.occupancy_grid_morton_bitfield, loader.nerf_network)
    buf = fvc.RenderBuffer((W, H))
    r.render(infos[0], buf)
    out += [buf.results.copy(), buf.ray_counts.copy()]
    res = torch.zeros((2 * W * H, 4), dtype=torch.float32, device="cuda")
    r.render_batch(infos, results=res)
    r.synchronize()
    out.append(res.cpu().numpy())
    one = torch.zeros((H, W, 4), dtype=torch.float32, device="cuda")
    o = L.RenderOutputs()
    o.results = one.data_ptr()
    L.check(L.load().fvc_render_noalloc(loader.nerf_network.handle, C.byref(infos[1]), C.byref(o), None))
    torch.cuda.synchronize()
    out.append(one.cpu().numpy())
    pred = torch.zeros((W * H, 4), dtype=torch.float32, device="cuda")
    r.render_backward(infos[0], torch.arange(W * H, dtype=torch.int32, device="cuda"), torch.zeros((W * H, 3), device="cuda"),
                      fvc.Gradients(loader.nerf_network), pred=pred)
    out.append(pred.cpu().numpy())
    for fill in ("initCacheBlockwise", "initCache"):
        c0, c1 = fvc.Cache(), fvc.Cache()
        rc = fvc.CachePerformanceRenderer(loader.scene_info, loader.occupancy_grid_morton_bitfield, loader.nerf_network, c0, c1)
        rc.resizeCache((W, H), steps)
        rc.resizeRenderbuffers((W, H))
        rc.setCacheSettings(fvc.default_cache_settings())
        getattr(rc, fill)(infos[0])
        out += [x.copy() for x in c1.read()[:2]]
        rc.swapCache()
        rc.render(infos[1], buf)
        out.append(buf.results.copy())
    return out


def test_edited_bits_are_seen(pair):
    torch = pytest.importorskip("torch")
    a, b = pair
    before, want = _everything(a, torch), _everything(b, torch)
    assert not all(np.array_equal(x, y) for x, y in zip(before, want))
    kept = _bits(a).clone()
    for bits, ref in ((_bits(b), want), (kept, before)):
        _bits(a).copy_(bits)
        torch.cuda.synchronize()
        for k, (x, y) in enumerate(zip(_everything(a, torch), ref)):
            np.testing.assert_array_equal(x.view(np.uint32), y.view(np.uint32), err_msg=str(k))


def test_a_captured_batch_sees_them(pair):
    """The batch's graph is built once and launched again."""
    torch = pytest.importorskip("torch")
    a, b = pair
    infos = [fvc.raymarch_info(small_camera(1601 + v, W, H), a.stepsize_info) for v in range(2)]
    res = torch.zeros((2 * W * H, 4), dtype=torch.float32, device="cuda")

    def batch(r):
        r.render_batch(infos, results=res)
        r.synchronize()
        return res.cpu().numpy().view(np.uint32)

    ra, rb = (fvc.PerformanceRenderer(x.scene_info, x.occupancy_grid_morton_bitfield, x.nerf_network) for x in (a, b))
    before, want = batch(ra), batch(rb)
    _bits(a).copy_(_bits(b))
    torch.cuda.synchronize()
    np.testing.assert_array_equal(batch(ra), want)
    assert not np.array_equal(before, want)
