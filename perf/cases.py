"""Performance cases: what a program on this renderer has it do, through the public Python API.

Scenes are the package's seeded synthetic models: "box" is the plain 256x256
workload's (one cascade over [-1.5, 1.5]^3, fixed steps), "unbounded" the
1080p camera path's (three cascades over [-6, 6]^3 with the L-infinity
contraction, steps that grow with distance).  Their random density is a fog
that no ray ever leaves early; "solid" scales the density output so that the
occupied cells are nearly opaque, as a trained scene's are, and rays end at
different depths.  A program loads its model once and renders many cameras
from it, so a model is loaded once per process and the seed picks the
cameras, pixels, targets and points.

exact() evaluates the same samples in float64: the step sequence, occupancy
test and sample positions are the method's float32 index arithmetic, the
network and the compositing are float64 without rounding between layers.
The cached renders have none: what they return depends on the fp16 voxels and
the slots of the cache.
"""
import atexit
import functools
import math
import os
import shutil
import tempfile
from dataclasses import replace

import numpy as np
import torch

import frustumvolumecaching_gb300 as fvc
from frustumvolumecaching_gb300 import camera as fcam
from frustumvolumecaching_gb300 import model as fmodel

DEV = "cuda"
#: mean samples a ray composites, by scene and solid, for work()
SAMPLES = {("box", False): 85, ("unbounded", False): 80, ("box", True): 28, ("unbounded", True): 35}
FLOP_SAMPLE = 16896  # density 2 * (32*64 + 64*9) + color 2 * (24*64 + 64*64 + 64*3)
PRECISIONS = {"fp16": 0, "bf16": 1, "fp8": 2}


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # a thumbnail or a drag preview: latency and launches
        {"name": "view_64", "do": "view", "w": 64, "h": 64, "scene": "box", "log2_T": 16, "solid": False, "precision": "fp16"},
        # the plain 256x256 workload
        {"name": "view_256", "do": "view", "w": 256, "h": 256, "scene": "box", "log2_T": 16, "solid": False, "precision": "fp16"},
        # the precision option, at a size that is no multiple of any tile
        {"name": "view_bf16", "do": "view", "w": 333, "h": 217, "scene": "box", "log2_T": 16, "solid": False, "precision": "bf16"},
        # a plain frame of the 1080p camera path
        {"name": "view_1080", "do": "view", "w": 1920, "h": 1080, "scene": "unbounded", "log2_T": 19, "solid": False, "precision": "fp16"},
        # an evaluation image of a scene with opaque surfaces, through host buffers
        {"name": "eval_solid", "do": "host", "w": 1283, "h": 717, "scene": "unbounded", "log2_T": 19, "solid": True, "precision": "fp16"},
        # a frame of the 1080p camera path with the frustum cache rebuilt, as each of its frames is
        {"name": "cached_1080", "do": "cached", "w": 1920, "h": 1080, "scene": "unbounded", "log2_T": 19, "solid": False, "fill": "blocks"},
        # the same at a preview window's size
        {"name": "cached_preview", "do": "cached", "w": 323, "h": 181, "scene": "unbounded", "log2_T": 19, "solid": False, "fill": "blocks"},
        # the per-ray cache fill and a frame from it, opaque surfaces
        {"name": "cached_rays", "do": "cached", "w": 640, "h": 360, "scene": "box", "log2_T": 16, "solid": True, "fill": "rays"},
        # several views of different sizes in one graph launch
        {"name": "batch_views", "do": "batch", "w": 960, "h": 540, "views": 8, "scene": "box", "log2_T": 16, "solid": False},
        # a training step of the differentiable workload: 2^18 random rays of an 800x800 view
        {"name": "train_2e18", "do": "train", "w": 800, "h": 800, "rays": 1 << 18, "scene": "box", "log2_T": 19, "solid": False, "precision": "fp16"},
        # a small training step on a small model, bf16 layers
        {"name": "train_small", "do": "train", "w": 200, "h": 200, "rays": 4099, "scene": "box", "log2_T": 16, "solid": False, "precision": "bf16"},
        # network queries from host arrays: density grids, probes
        {"name": "query_points", "do": "query", "points": 1 << 19, "scene": "unbounded", "log2_T": 19, "solid": False},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    do = rng.choice(["view", "view", "view", "host", "cached", "cached", "batch", "train", "train", "query"])
    scene = rng.choice(["box", "unbounded"])
    c = {"do": do, "scene": scene, "log2_T": rng.choice([16, 19]), "solid": rng.random() < 0.4}
    if do == "query":
        return c | {"points": _log_int(rng, 1, 1 << 19)}
    if do == "train":
        side = _log_int(rng, 64, 800)
        return c | {"scene": "box", "w": side, "h": side, "rays": _log_int(rng, 256, min(side * side, 1 << 18)), "precision": rng.choice(["fp16", "bf16"])}
    w = _log_int(rng, 48, 1920)
    c |= {"w": w, "h": max(17, round(w * rng.uniform(0.5, 0.5625)))}
    if do == "batch":
        return c | {"w": max(96, w // 2), "h": max(64, c["h"] // 2), "views": rng.randint(2, 8)}
    if do == "cached":
        return c | {"fill": rng.choice(["blocks", "blocks", "rays"])}
    return c | {"precision": rng.choice(["fp16", "fp16", "bf16", "fp8"])}


# ---------------------------------------------------------------------------
# models
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _parameters(scene, log2_T, solid):
    """The synthetic model's parameters and occupancy grid."""
    spec = replace(fmodel.spec_config1() if scene == "box" else fmodel.spec_config2(), log2_T=log2_T)
    sm = fmodel.SyntheticModel(spec)
    net = _Net64(sm, dtype=torch.float32)
    occ, inside = [], []
    for level in range(spec.grid_nlvl):
        p = fmodel.contract(sm.cell_centres_world(level), sm.scene_dict())
        ld = torch.cat([net.density(q)[:, 0] for q in torch.from_numpy(p).to(DEV, torch.float32).split(1 << 20)])
        k = int(ld.numel() * (1.0 - spec.occupancy_fraction))
        thr = ld.kthvalue(k).values
        occ.append((ld > thr).to(torch.uint8).cpu().numpy())
        inside.append(ld[ld > thr].median())
    sm.occupancy = np.concatenate(occ)
    if solid:  # the median occupied cell at density e^4.5: a ray ends within a few hundredths of a unit
        k = 4.5 / float(torch.stack(inside).mean())
        sm.base[1][0] = (sm.base[1][0].astype(np.float32) * k).astype(np.float16)
    return sm


@functools.lru_cache(maxsize=None)
def _root():
    d = tempfile.mkdtemp(prefix="fvc_cases_")
    atexit.register(shutil.rmtree, d, True)
    return d


@functools.lru_cache(maxsize=None)
def _loaded(scene, log2_T, solid):
    d = os.path.join(_root(), f"{scene}_{log2_T}_{int(solid)}")
    _parameters(scene, log2_T, solid).write(d)
    data = fvc.load_data(d)
    shutil.rmtree(d, True)
    return data


def _key(case):
    return case["scene"], case["log2_T"], case["solid"]


def _renderer(cls, data, *caches):
    return cls(data.scene_info, data.occupancy_grid_morton_bitfield, data.nerf_network, *caches)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _camera(seed, w, h):
    return fcam.seeded_camera(int(seed) * 7919 + 11, width=w, height=h)


def _next_camera(seed, w, h):
    """The camera path's next frame: half a degree around the up axis."""
    return fcam.rotation_path(int(seed) * 7919 + 11, n_frames=2, width=w, height=h)[1]


def _view_sizes(case):
    """Views of a batch have the case's size and fractions of it."""
    return [(max(8, int(case["w"] * f)), max(8, int(case["h"] * f))) for f in (1.0, 2 / 3, 1 / 3, 1 / 6) * 2][: case["views"]]


def _batch_cameras(case, seed):
    return [_camera(int(seed) * 64 + v, w, h) for v, (w, h) in enumerate(_view_sizes(case))]


def _pixels(case, seed):
    rng = np.random.default_rng([int(seed), 5])
    pix = rng.choice(case["w"] * case["h"], case["rays"], replace=False).astype(np.int32)
    # targets: a smooth picture with noise
    x, y = (pix % case["w"]) / case["w"], (pix // case["w"]) / case["h"]
    base = 0.5 + 0.3 * np.stack([np.sin(7 * x + 3 * y), np.cos(5 * y - 2 * x), np.sin(9 * x * y + 1)], axis=1)
    return pix, np.clip(base + rng.normal(0, 0.05, base.shape), 0, 1).astype(np.float32)


def _points(case, seed):
    rng = np.random.default_rng([int(seed), 6])
    d = rng.normal(size=(case["points"], 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return rng.random((case["points"], 3), dtype=np.float32), ((d + 1.0) / 2.0).astype(np.float32)


class State:
    pass


def prepare(case, seed):
    s = State()
    s.do = case["do"]
    data = _loaded(*_key(case))
    steps = data.stepsize_info
    if s.do == "query":
        s.net = data.nerf_network
        s.pos, s.dir01 = _points(case, seed)
        return s
    if s.do == "batch":
        cams = _batch_cameras(case, seed)
        s.infos = [fvc.raymarch_info(c, steps) for c in cams]
        s.renderer = _renderer(fvc.PerformanceRenderer, data)
        n = sum(c["resolution"][0] * c["resolution"][1] for c in cams)
        s.renderer.resizeRenderbuffers((n, 1))
        s.results = torch.zeros((n, 4), dtype=torch.float32, device=DEV)
        return s
    w, h = case["w"], case["h"]
    s.info = fvc.raymarch_info(_camera(seed, w, h), steps)
    if s.do == "train":
        pix, target = _pixels(case, seed)
        s.pixels, s.target = torch.from_numpy(pix).to(DEV), torch.from_numpy(target).to(DEV)
        s.pred = torch.zeros((case["rays"], 4), dtype=torch.float32, device=DEV)
        s.grads = fvc.Gradients(data.nerf_network)
        s.renderer = _renderer(fvc.PerformanceRenderer, data)
        s.renderer.set_precision(PRECISIONS[case["precision"]])
        s.renderer.resizeRenderbuffers((w, h))
        return s
    if s.do == "cached":
        s.renderer = _renderer(fvc.CachePerformanceRenderer, data, fvc.Cache(), fvc.Cache())
        for _ in range(2):  # both caches of the pair
            s.renderer.resizeCache((w, h), steps)
            s.renderer.swapCache()
        s.renderer.resizeRenderbuffers((w, h))
        s.build = s.renderer.initCacheBlockwise if case["fill"] == "blocks" else s.renderer.initCache
        s.next_info = fvc.raymarch_info(_next_camera(seed, w, h), steps)
    else:
        s.renderer = _renderer(fvc.PerformanceRenderer, data)
        s.renderer.set_precision(PRECISIONS[case["precision"]])
        s.renderer.resizeRenderbuffers((w, h))
    if s.do == "host":
        s.buffer = fvc.RenderBuffer((w, h))
    else:
        s.results = torch.zeros((h, w, 4), dtype=torch.float32, device=DEV)
        s.image = torch.zeros((h, w, 4), dtype=torch.uint8, device=DEV)
    return s


def run(s):
    if s.do == "query":
        return {"logits": s.net.inference(s.pos, s.dir01)}
    if s.do == "batch":
        s.renderer.render_batch(s.infos, results=s.results)
        return {"results": s.results}
    if s.do == "train":
        s.grads.zero()
        loss = s.renderer.render_backward(s.info, s.pixels, s.target, s.grads, pred=s.pred)
        table, base, head = s.grads.read()
        return {"loss": loss, "pred": s.pred, "table": table, "base": base, "head": head}
    if s.do == "host":
        s.renderer.render(s.info, s.buffer)
        return {"results": s.buffer.results, "image": s.buffer.image, "counts": s.buffer.ray_counts}
    if s.do == "cached":
        s.build(s.info)
        s.renderer.swapCache()
        s.renderer.render_device(s.next_info, image=s.image, results=s.results)
    else:
        s.renderer.render_device(s.info, image=s.image, results=s.results)
    return {"results": s.results, "image": s.image}


def work(case):
    """What no implementation can do without: the parameters and occupancy
    read once, the outputs written once, and the networks of the occupied
    samples (a cached frame's network work is that of a plain frame)."""
    sm = fmodel.hash_grid_levels(16, 16, 1.447, case["log2_T"])
    table = 4 * (sm[-1].offset + sm[-1].size)
    model = table + 128 ** 3 // 8 * (1 if case["scene"] == "box" else 3) + 20480
    if case["do"] == "query":
        return {"bytes": table + 40 * case["points"], "flops": FLOP_SAMPLE * case["points"]}
    if case["do"] == "train":
        rays = case["rays"]  # the adjoint is twice the forward's contractions
        return {"bytes": model + 2 * table + 32 * rays, "flops": 3 * FLOP_SAMPLE * SAMPLES["box", case["solid"]] * rays}
    if case["do"] == "batch":
        rays, out = sum(w * h for w, h in _view_sizes(case)), 16
    else:
        rays, out = case["w"] * case["h"], 36 if case["do"] == "host" else 20
    return {"bytes": model + out * rays, "flops": FLOP_SAMPLE * SAMPLES[case["scene"], case["solid"]] * rays}


# ---------------------------------------------------------------------------
# the same in float64
# ---------------------------------------------------------------------------
class _Net64:
    """The hash grid, density network and color head in plain torch."""

    def __init__(self, sm, dtype=torch.float64):
        def t(a):
            return torch.from_numpy(np.asarray(a, np.float32)).to(DEV, dtype)
        self.spec, self.levels, self.dtype = sm.spec, sm.levels, dtype
        self.table = t(sm.table)
        self.base, self.head = [t(w) for w in sm.base], [t(w) for w in sm.head]

    def features(self, pos):
        p32, out = pos.float(), []
        for lv in self.levels:
            # the cell and the fraction of the float32 point fma(scale, x, 0.5)
            p = (p32.double() * float(np.float32(lv.scale)) + 0.5).float()
            g = p.floor()
            f = (p - g).to(self.dtype)
            g = g.long()
            acc = None
            for c in range(8):
                ix, iy, iz = g[:, 0] + (c & 1), g[:, 1] + ((c >> 1) & 1), g[:, 2] + (c >> 2)
                if lv.dense:
                    i = (ix + iy * lv.res + iz * lv.res ** 2) % lv.size
                else:
                    i = (ix ^ (iy * 2654435761) ^ (iz * 805459861)) & (lv.size - 1)
                w = ((f[:, 0] if c & 1 else 1 - f[:, 0]) * (f[:, 1] if c & 2 else 1 - f[:, 1]) * (f[:, 2] if c & 4 else 1 - f[:, 2]))
                v = w[:, None] * self.table[i + lv.offset]
                acc = v if acc is None else acc + v
            out.append(acc)
        return torch.cat(out, 1)

    def density(self, pos):
        return torch.relu(self.features(pos) @ self.base[0].T) @ self.base[1].T

    def color(self, latents, d):
        x, y, z = d.to(self.dtype).unbind(1)
        x2, y2, z2 = x * x, y * y, z * z
        c = _sh_constants()
        sh = [torch.full_like(x, c["c0"]), -c["c1"] * y, c["c1"] * z, -c["c1"] * x, c["c2a"] * x * y, -c["c2a"] * y * z, c["c2b"] * (3 * z2 - 1),
              -c["c2a"] * x * z, c["c2c"] * (x2 - y2), c["c3a"] * y * (-3 * x2 + y2), c["c3b"] * x * y * z, c["c3c"] * y * (1 - 5 * z2),
              c["c3d"] * z * (5 * z2 - 3), c["c3c"] * x * (1 - 5 * z2), c["c3e"] * z * (x2 - y2), c["c3a"] * x * (-x2 + 3 * y2)]
        h = torch.cat([latents, torch.stack(sh, 1), torch.ones((len(x), 8), dtype=self.dtype, device=DEV)], 1)  # padded with ones
        for w in self.head[:-1]:
            h = torch.relu(h @ w.T)
        return (h @ self.head[-1].T)[:, :3]


def _sh_constants():
    """Real spherical harmonics to degree 3: the constants of each band."""
    s, pi = math.sqrt, math.pi
    return {"c0": 1 / (2 * s(pi)), "c1": s(3) / (2 * s(pi)), "c2a": s(15) / (2 * s(pi)), "c2b": s(5) / (4 * s(pi)), "c2c": s(15) / (4 * s(pi)),
            "c3a": s(70) / (8 * s(pi)), "c3b": s(105) / (2 * s(pi)), "c3c": s(42) / (8 * s(pi)), "c3d": s(7) / (4 * s(pi)), "c3e": s(105) / (4 * s(pi))}


def _f32(*v):
    return [torch.tensor(np.float32(x), device=DEV) for x in v]


def _rays(cam, px, py):
    """Pixel-centre rays in float32."""
    m = torch.from_numpy(np.asarray(cam["cam2world"], np.float32)).to(DEV)
    (fx, fy), (cx, cy) = _f32(*cam["focal"]), _f32(*cam["principal"])
    x, y = (px.float() + 0.5 - cx) / fx, (py.float() + 0.5 - cy) / fy
    v = torch.stack([x * m[r, 0] + y * m[r, 1] + m[r, 2] for r in range(3)], 1)
    inv = (1.0 / ((v[:, 0] * v[:, 0] + v[:, 1] * v[:, 1]) + v[:, 2] * v[:, 2]).double().sqrt()).float()
    return m[:, 3].expand_as(v), v * inv[:, None]


def _samples(sm, cam, px, py):
    """The occupied samples of each ray: (ray, number in the ray, distance, step, position), and the ray directions."""
    s = sm.spec
    o, d = _rays(cam, px, py)
    lo, hi = (torch.tensor(v, dtype=torch.float32, device=DEV) for v in (s.aabb[:3], s.aabb[3:]))
    a, b = (lo - o) / d, (hi - o) / d
    near, far = torch.minimum(a, b).amax(1), torch.maximum(a, b).amin(1)
    hits = near <= far
    step = np.float32(s.stepsize)
    extent = max(np.float32(s.aabb[3 + k]) - np.float32(s.aabb[k]) for k in range(3))
    dt_max = np.float32(np.float32(extent) / np.float32(128) * np.float32(1.732))
    cone = np.float32(s.cone_angle)
    t = near.clamp(min=s.near).double()
    if cone > 0:
        t_min, i_min, lg = float(step) / float(cone), 1.0 / float(cone), math.log1p(float(cone))
        i_max = math.log(float(dt_max) / float(step)) / lg + i_min
        t_max = t_min * math.exp(lg * (i_max - i_min))
        i = torch.where(t >= t_max, (t - t_max) / float(dt_max) + i_max, torch.where(t < t_min, t / float(step), torch.log(t / t_min) / lg + i_min))
        i = torch.floor(i + 0.5)
        t = torch.where(i >= i_max, t_max + (i - i_max) * float(dt_max), torch.where(i < i_min, i * float(step), t_min * torch.exp(lg * (i - i_min))))
    else:
        t = torch.floor(t / float(step) + 0.5) * float(step)
    t = t.float()
    step, dt_max, cone = _f32(step, dt_max, cone)
    scale = 2.0 ** (s.grid_nlvl - 1)
    off, den = lo / scale, hi / scale - lo / scale
    occ = torch.from_numpy(sm.occupancy).to(DEV).view(s.grid_nlvl, -1)
    alive, count, rows = hits.clone(), torch.zeros(len(t), dtype=torch.long, device=DEV), []
    it = 0
    while it % 16 or bool(alive.any()):
        it += 1
        dt = torch.maximum(step, torch.minimum(t * cone, dt_max))
        t1 = t + dt
        tm = (t + t1) * 0.5
        alive = alive & (tm <= far)
        p = o + tm[:, None] * d
        u = (p - off) / den - 0.5
        mip = torch.frexp(u.abs().amax(1))[1].add(1).clamp(min=0)
        cell = ((u * torch.exp2(-mip.float())[:, None] + 0.5) * 128).long().clamp(0, 127)
        on = occ[mip.clamp(max=s.grid_nlvl - 1), cell[:, 0] * 16384 + cell[:, 1] * 128 + cell[:, 2]] > 0
        r = (alive & (mip < s.grid_nlvl) & on).nonzero()[:, 0]
        rows.append((r, count[r], t[r], dt[r], p[r]))
        count[r] += 1
        t = t1
    ray, k, t0, dt, p = (torch.cat(v) for v in zip(*rows))
    p = p.double()
    if s.contraction == "linf":
        c = torch.tensor(s.contraction_aabb, dtype=torch.float64, device=DEV)
        u = (p - c[:3]) / (c[3:] - c[:3]) * 2 - 1
        f = u.abs().amax(1, keepdim=True).clamp(min=1.0)
        p = (2 - 1 / f) * (u / f) / 4 + 0.5
    else:
        p = (p - lo.double()) / (hi - lo).double()
    return ray, k, t0, dt, p, d


def _composite(n, ray, k, dt, log_density, logits):
    """Front to back: colour and transmittance of n rays, ended below a transmittance of 1e-4."""
    width = int(k.max()) + 1 if len(k) else 1
    at = ray * width + k
    alpha = 1 - torch.exp(-torch.exp(log_density) * dt.double())
    grid = torch.zeros(n * width, dtype=torch.float64, device=DEV).index_put((at,), alpha).view(n, width)
    after = torch.cumprod(1 - grid, 1)
    before = torch.cat([torch.ones((n, 1), dtype=torch.float64, device=DEV), after[:, :-1]], 1)
    live = before.detach() >= 1e-4
    w = (grid * before * live).reshape(-1)[at]
    color = torch.zeros((n, 3), dtype=torch.float64, device=DEV).index_add(0, ray, w[:, None] * torch.sigmoid(logits))
    left = torch.where(live, 1 - grid, 1.0).prod(1)
    return torch.cat([color, left[:, None]], 1)


def _network(net, pos, d, ray):
    out = net.density(pos)
    return out[:, 0], net.color(out[:, 1:9], d[ray])


def _image64(sm, net, cam):
    w, h = cam["resolution"]
    out = torch.empty((h * w, 4), dtype=torch.float64, device=DEV)
    for pix in torch.arange(h * w, device=DEV).split(1 << 18):
        ray, k, _, dt, p, d = _samples(sm, cam, pix % w, pix // w)
        got = [_network(net, q, d, r) for q, r in zip(p.split(1 << 21), ray.split(1 << 21))]
        ld, lg = (torch.cat(v) for v in zip(*got))
        out[pix] = _composite(len(pix), ray, k, dt, ld, lg)
    return out.view(h, w, 4)


def _train64(sm, net, cam, pix, target):
    params = [net.table, *net.base, *net.head]
    for v in params:
        v.requires_grad_(True)
    pred, loss = torch.empty((len(pix), 4), dtype=torch.float64, device=DEV), 0.0
    pix, target = torch.from_numpy(pix).to(DEV).long(), torch.from_numpy(target).to(DEV, torch.float64)
    w = cam["resolution"][0]
    for at in torch.arange(len(pix), device=DEV).split(1 << 13):
        with torch.no_grad():
            ray, k, _, dt, p, d = _samples(sm, cam, pix[at] % w, pix[at] // w)
        ld, lg = _network(net, p, d, ray)
        out = _composite(len(at), ray, k, dt, ld, lg)
        part = (out[:, :3] + out[:, 3:] - target[at]).square().sum() / len(pix)
        if part.requires_grad and len(ray):
            part.backward()
        pred[at] = out.detach()
        loss += float(part.detach())
    grads = [v.grad.reshape(-1) if v.grad is not None else torch.zeros(v.numel(), dtype=torch.float64, device=DEV) for v in params]
    n = 1 + len(net.base)
    return {"loss": loss, "pred": pred, "table": grads[0], "base": torch.cat(grads[1:n]), "head": torch.cat(grads[n:])}


def exact(case, seed):
    if case["do"] == "cached":
        return None
    sm = _parameters(*_key(case))
    net = _Net64(sm)
    if case["do"] == "train":
        pix, target = _pixels(case, seed)
        return _train64(sm, net, _camera(seed, case["w"], case["h"]), pix, target)
    with torch.no_grad():
        if case["do"] == "query":
            pos, dir01 = (torch.from_numpy(a).to(DEV) for a in _points(case, seed))
            ld, lg = _network(net, pos, dir01.double() * 2 - 1, torch.arange(len(pos), device=DEV))
            return {"logits": torch.cat([lg, ld[:, None]], 1)}
        if case["do"] == "batch":
            return {"results": torch.cat([_image64(sm, net, c).view(-1, 4) for c in _batch_cameras(case, seed)])}
        img = _image64(sm, net, _camera(seed, case["w"], case["h"]))
        return {"results": img, "image": None, "counts": None} if case["do"] == "host" else {"results": img, "image": None}
