"""The work that users have this renderer do, as measurable cases.

Every case goes through the public Python entry points of `yoxel`, on seeded
synthetic scenes made on the GPU (the reference ships no scene data):

  svo      one frame of an octree: first hit, Lambert, optional shadow rays
  lod      the same with the level-of-detail cut-off, on by default in CudaRenderer
  edit     an interactive edit: recolour voxels, sync the changed pages, redraw
  ssna     a frame shaded by screen-space normals and a point light
  brick    brick volume composites of one or several cameras
  train    forward and backward of the differentiable march (inverse rendering)
  batch    many small scenes of both types in one launch (thumbnails, views)
  svolive  a new dense field each frame: build the octree, draw it
  volive   a new dense lattice each frame: rebuild the brick pool, draw it
"""
import math
import os
import random
import sys

import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "yoxel-voxel_gb300"))
import yoxel  # noqa: E402
from yoxel import _lib  # noqa: E402

LIGHT = tuple(v / math.sqrt(0.3 ** 2 + 0.5 ** 2 + 0.8 ** 2) for v in (0.3, 0.5, 0.8))
FOV = 60.0
FITTED = 77  # the bricks of the volumes that are fitted
F16, F32, F16_PACKED = _lib.YV_PRECISION_F16, _lib.YV_PRECISION_F32, _lib.YV_PRECISION_F16_PACKED


def listed():
    return [
        # a thumbnail or the first preview while the camera moves: latency and launches
        dict(name="svo_preview", kind="svo", scene="spheres", depth=8, width=160, height=120,
             shadows=False),
        # the flagship frame: a 2048^3 landscape at full HD with a shadow ray per hit
        dict(name="svo_terrain_1080p", kind="svo", scene="terrain", depth=11, width=1920,
             height=1080, shadows=True),
        # the Python driver's default window with its detail cut-off, odd by a pixel
        dict(name="lod_window", kind="lod", scene="spheres", depth=9, width=641, height=479,
             detail=4.0),
        # painting on a 256^3 model: a brush stroke, page sync, redraw
        dict(name="edit_paint", kind="edit", scene="spheres", depth=8, width=512, height=512,
             edits=64),
        # the demo viewer's shading at full HD
        dict(name="ssna_1080p", kind="ssna", scene="terrain", depth=10, width=1920, height=1080),
        # a 512^3 scan in the compact pool, one large frame
        dict(name="brick_scan", kind="brick", levels=3, precision=F16_PACKED, cams=1, width=1024,
             height=1024, step=0.5),
        # a turntable of a 128^3 volume: several ragged frames, separate fp16 / RGB arrays
        dict(name="brick_turntable", kind="brick", levels=2, precision=F16, cams=7, width=333,
             height=251, step=0.5),
        # one small step of fitting a volume to a few views (a debugging or coarse stage)
        dict(name="train_coarse", kind="train", levels=2, cams=4, width=64, height=64),
        # the fitting step: 64 views at 256^2 of a 128^3 volume, forward and backward
        dict(name="train_views", kind="train", levels=2, cams=64, width=256, height=256),
        # mixed requests of a render service answered in one launch
        dict(name="batch_mixed", kind="batch", scenes=16, mix=5, most=1024),
        # a 1024^3 simulated field drawn as an octree each step
        dict(name="svo_live", kind="svolive", scene="spheres", depth=10, width=512, height=512),
        # a 512^3 simulated lattice drawn as a brick volume each step, as an 8-bit image
        dict(name="volume_live", kind="volive", levels=3, precision=F16_PACKED, width=512,
             height=512),
    ]


def _size(rng, lo, hi):
    """A size spread over its logarithm, odd ones among them."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["svo", "svo", "lod", "edit", "ssna", "brick", "brick", "train", "train",
                       "batch", "svolive", "volive"])
    w, h = _size(rng, 96, 1900), _size(rng, 72, 1080)
    if kind == "svo":
        return dict(kind=kind, scene=rng.choice(["spheres", "terrain"]), depth=rng.randint(6, 10),
                    width=w, height=h, shadows=rng.random() < 0.5)
    if kind == "lod":
        return dict(kind=kind, scene="spheres", depth=rng.randint(7, 9), width=w, height=h,
                    detail=rng.choice([1.0, 2.0, 4.0, 8.0]))
    if kind == "edit":
        return dict(kind=kind, scene="spheres", depth=rng.randint(6, 8), width=w, height=h,
                    edits=_size(rng, 8, 200))
    if kind == "ssna":
        return dict(kind=kind, scene="terrain", depth=rng.randint(8, 10), width=w, height=h)
    if kind == "brick":
        levels = rng.choice([1, 2, 3])
        return dict(kind=kind, levels=levels, precision=rng.choice([F16, F32, F16_PACKED]),
                    cams=1 if levels == 3 else rng.randint(1, 9), width=min(w, 1024),
                    height=min(h, 1024), step=rng.choice([0.5, 0.5, 1.0, 0.37]))
    if kind == "train":
        s = _size(rng, 48, 256)
        return dict(kind=kind, levels=rng.choice([1, 2, 2]), cams=_size(rng, 1, 60), width=s,
                    height=max(32, s - rng.randint(0, 15)))
    if kind == "batch":
        return dict(kind=kind, scenes=rng.randint(4, 24), mix=rng.randrange(1000),
                    most=rng.choice([256, 512]))
    if kind == "svolive":
        return dict(kind=kind, scene=rng.choice(["spheres", "terrain"]), depth=rng.randint(6, 9),
                    width=min(w, 1024), height=min(h, 1024))
    return dict(kind=kind, levels=rng.choice([1, 2, 3]),
                precision=rng.choice([F16, F32, F16_PACKED]), width=min(w, 700),
                height=min(h, 700))


# ---- seeded inputs ------------------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFF)


def _spheres(depth, seed):
    """Signed field of 200 spheres (radii 4..24 voxels of a 256^3 grid, scaled), > 0 inside."""
    G = 1 << depth
    f = torch.full((G, G, G), -1.0, device="cuda")
    r = random.Random(seed * 7919 + 13)
    ax = torch.arange(G, device="cuda", dtype=torch.float32) + 0.5
    for _ in range(200):
        c = [r.uniform(0.1, 0.9) * G for _ in range(3)]
        rad = r.uniform(4.0, 24.0) * G / 256.0
        s = [slice(max(0, int(v - rad) - 2), min(G, int(v + rad) + 3)) for v in c]
        d2 = ((ax[s[2]] - c[2]) ** 2)[:, None, None] + ((ax[s[1]] - c[1]) ** 2)[None, :, None] + \
            ((ax[s[0]] - c[0]) ** 2)[None, None, :]
        sub = f[s[2], s[1], s[0]]
        torch.maximum(sub, rad - d2.sqrt_(), out=sub)
    return f


def _octaves2(G, g):
    """Value noise in [-1, 1]: 6 octaves of bicubic lattices, spacing G/8 down."""
    h = torch.zeros((G, G), device="cuda")
    w, tot = 1.0, 0.0
    for o in range(6):
        n = min(G, (8 << o) + 1)
        t = torch.rand((1, 1, n, n), generator=g, device="cuda") * 2 - 1
        h += w * torch.nn.functional.interpolate(t, size=(G, G), mode="bicubic",
                                                 align_corners=True)[0, 0]
        tot += w
        w *= 0.5
    return h / tot


def _terrain(depth, seed):
    """A landscape below a height field, with a few hundred floating blocks."""
    G = 1 << depth
    h = G * (0.5 + 0.3 * _octaves2(G, _gen(seed)))
    f = torch.empty((G, G, G), device="cuda")
    z = torch.arange(G, device="cuda", dtype=torch.float32)
    torch.sub(h[None], z[:, None, None], out=f)
    r = random.Random(seed * 104729 + 7)
    for _ in range(400):
        s = r.randint(2, 16)
        x, y, k = (r.randrange(max(1, G - s)) for _ in range(3))
        f[k:k + s, y:y + s, x:x + s] = 1.0
    return f


def _field(case, seed):
    return (_spheres if case["scene"] == "spheres" else _terrain)(case["depth"], seed)


def _paint(depth, seed):
    """RGB of every voxel: smooth colours (none above 512^3, where white is used)."""
    if depth > 9:
        return None
    G = 1 << depth
    t = torch.rand((1, 3, 9, 9, 9), generator=_gen(seed + 1), device="cuda")
    t = torch.nn.functional.interpolate(t, size=(G, G, G), mode="trilinear", align_corners=True)
    return (t[0] * 255).to(torch.uint8).permute(1, 2, 3, 0).contiguous()


def _lattice(levels, seed, shape=None):
    """Density in [0, 1], zero in most of the volume, and RGB, on the (8 4^levels + 1)^3 lattice.

    shape: a seed of its own for where the density is not zero (a volume that is being fitted
    keeps its bricks)."""
    n = 8 * 4 ** levels + 1
    g = _gen(seed + 2 if shape is None else shape)
    f = torch.zeros((1, 1, n, n, n), device="cuda")
    w, tot = 1.0, 0.0
    for o in range(4):
        m = min(n, (8 << o) + 1)
        t = torch.rand((1, 1, m, m, m), generator=g, device="cuda") * 2 - 1
        f += w * torch.nn.functional.interpolate(t, size=(n, n, n), mode="trilinear",
                                                 align_corners=True)
        tot += w
        w *= 0.5
    density = (f[0, 0] * (2.6 / tot) - 0.55).clamp_(0.0, 1.0).contiguous()
    if shape is not None:
        g = _gen(seed + 2)
        t = torch.rand((1, 1, 17, 17, 17), generator=g, device="cuda") * 0.8 + 0.2
        density *= torch.nn.functional.interpolate(t, size=(n, n, n), mode="trilinear",
                                                   align_corners=True)[0, 0]
    t = torch.rand((1, 3, 17, 17, 17), generator=g, device="cuda")
    t = torch.nn.functional.interpolate(t, size=(n, n, n), mode="trilinear", align_corners=True)
    return density, (t[0] * 255).to(torch.uint8).permute(1, 2, 3, 0).contiguous()


def _camera(seed, k=0):
    """A camera around the scene centre, 1.5 scene sides away, looking at it."""
    r = random.Random(seed * 31 + k * 1009 + 5)
    d = [1.0 + r.uniform(-0.2, 0.2), 0.7 + r.uniform(-0.2, 0.2), 0.5 + r.uniform(-0.2, 0.2)]
    if k:
        a = 2.399963 * k
        d = [math.cos(a), math.sin(a), r.uniform(-0.6, 0.8)]
    n = math.sqrt(sum(v * v for v in d))
    d = [v / n for v in d]
    f32 = torch.tensor([0.5 + 1.5 * v for v in d] + [-v for v in d], dtype=torch.float32).tolist()
    return f32[:3], f32[3:], (0.0, 0.0, 1.0), FOV


def _cameras(case, seed):
    n = case.get("cams", 1)
    return [_camera(seed, k if n > 1 else 0) for k in range(n)]


def _renderer(width, height, seed, shadows=False):
    r = yoxel.Renderer()
    pos, view, up, fov = _camera(seed)
    r.SetViewPos(pos)
    r.SetViewDir(view)
    r.SetViewUp(up)
    r.SetFOV(fov)
    r.SetResolution(width, height)
    r.SetLight(LIGHT, 0.15, 0.85, shadows)
    return r


def _frame(width, height):
    mk = dict(device="cuda")
    return dict(rgba=torch.empty((height, width), dtype=torch.int32, **mk),
                hit=torch.empty((height, width), dtype=torch.int32, **mk),
                hit_t=torch.empty((height, width), dtype=torch.float32, **mk))


def _batch_specs(case):
    r = random.Random(case["mix"])
    sizes = [s for s in (128, 256, 512, 1024) if s <= case["most"]]
    specs = []
    for i in range(case["scenes"]):
        svo = r.random() < 0.5 if i else True
        specs.append(dict(svo=svo, res=r.choice(sizes), depth=r.randint(6, 9),
                          levels=r.choice([1, 2, 2, 3]), odd=r.choice([0, 0, 3])))
    specs[1].update(svo=False, res=sizes[-1], levels=3)
    return specs


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("svo", "ssna", "svolive"):
        w, h = case["width"], case["height"]
        r = _renderer(w, h, seed, case.get("shadows", False))
        f, rgb = _field(case, seed), _paint(case["depth"], seed)
        s = dict(kind=kind, renderer=r, depth=case["depth"])
        if kind == "svolive":
            s.update(field=f, rgb=rgb, out=_frame(w, h))
            return s
        r.SetSceneDense(f, case["depth"], 0.0, rgb)
        if kind == "svo":
            s.update(out=_frame(w, h))
        else:
            s.update(params=r.ssna_params(),
                     rgba=torch.empty((h, w), dtype=torch.int32, device="cuda"),
                     depth=torch.empty((h, w), dtype=torch.float32, device="cuda"))
        return s
    if kind in ("lod", "edit"):
        w, h = case["width"], case["height"]
        r = _renderer(w, h, seed)
        f, rgb = _field(case, seed), _paint(case["depth"], seed)
        scene = yoxel.SVOScene.build_dense(f, case["depth"], 0.0, rgb)
        s = dict(kind=kind, renderer=r, depth=case["depth"], out=_frame(w, h))
        if kind == "lod":
            r.SetScene(scene.build_lod())
            r.SetDetailCoef(case["detail"])
            return s
        dyn = yoxel.DynamicSVO(scene.node_count + 4096, scene.attr_count + 4096)
        dyn.load(scene)
        dyn.sync()
        r.SetSceneDynamic(dyn)
        # the stroke: surface voxels in one column-major run, each a colour of its own
        solid = f > 0
        surf = solid.clone()
        surf[1:-1, 1:-1, 1:-1] &= ~(solid[2:, 1:-1, 1:-1] & solid[:-2, 1:-1, 1:-1] &
                                    solid[1:-1, 2:, 1:-1] & solid[1:-1, :-2, 1:-1] &
                                    solid[1:-1, 1:-1, 2:] & solid[1:-1, 1:-1, :-2])
        at = surf.nonzero()
        first = random.Random(seed).randrange(max(1, at.shape[0] - case["edits"]))
        rnd = random.Random(seed + 1)
        s.update(dyn=dyn, edits=[(x, y, z, tuple(rnd.randrange(256) for _ in range(3)))
                                 for z, y, x in at[first:first + case["edits"]].tolist()])
        return s
    if kind == "brick":
        d, rgb = _lattice(case["levels"], seed)
        vol = yoxel.VolumeGPU.from_dense(d, case["levels"], case["precision"], rgb)
        return dict(kind=kind, volume=vol, desc=vol.desc(), size=(case["width"], case["height"]),
                    step=case["step"], cams=yoxel.cameras(_cameras(case, seed)),
                    out=torch.empty((case["cams"], case["height"], case["width"], 4),
                                    device="cuda"))
    if kind == "train":
        d, rgb = _lattice(case["levels"], seed, FITTED)
        tv = yoxel.BrickVolume.build_dense(d, case["levels"], rgb).to_torch()
        g = torch.randn((case["cams"], case["height"], case["width"], 4), generator=_gen(seed + 3),
                        device="cuda")
        return dict(kind=kind, tv=tv, density=tv["density"].requires_grad_(True),
                    albedo=tv["albedo"].requires_grad_(True),
                    cams=yoxel.cameras(_cameras(case, seed)),
                    size=(case["width"], case["height"]), grad=g)
    if kind == "batch":
        b, out, keep = yoxel.Batch(), [], []
        for i, sp in enumerate(_batch_specs(case)):
            w, h = sp["res"] + sp["odd"], sp["res"]
            if sp["svo"]:
                r = _renderer(w, h, seed + i)
                f = _spheres(sp["depth"], seed + i)
                r.SetSceneDense(f, sp["depth"], 0.0, _paint(sp["depth"], seed + i))
                out.append(torch.empty((h, w), dtype=torch.int32, device="cuda"))
                b.add_svo(r, out[-1])
                keep.append(r)
            else:
                d, rgb = _lattice(sp["levels"], seed + i)
                v = yoxel.VolumeGPU.from_dense(d, sp["levels"], F16_PACKED, rgb)
                out.append(torch.empty((h, w, 4), device="cuda"))
                b.add_volume(v.desc(), _camera(seed + i), w, h, out[-1])
                keep.append(v)
        return dict(kind=kind, batch=b, out=out, keep=keep)
    if kind == "volive":
        d, rgb = _lattice(case["levels"], seed)
        vol = yoxel.VolumeGPU.from_dense(d, case["levels"], case["precision"], rgb)
        return dict(kind=kind, volume=vol, density=d, rgb=rgb, levels=case["levels"],
                    size=(case["width"], case["height"]), cams=yoxel.cameras([_camera(seed)]),
                    out=torch.empty((1, case["height"], case["width"]), dtype=torch.int32,
                                    device="cuda"))
    raise ValueError(kind)


# ---- one pass -----------------------------------------------------------------------------

def run(s):
    kind = s["kind"]
    if kind in ("svo", "lod"):
        s["renderer"].render_async(**s["out"])
        return s["out"]
    if kind == "edit":
        for x, y, z, rgb in s["edits"]:
            s["dyn"].set_voxel(s["depth"], x, y, z, rgb)
        s["dyn"].sync()
        s["renderer"].render_async(**s["out"])
        return s["out"]
    if kind == "ssna":
        s["renderer"].render_ssna(s["params"], s["rgba"], s["depth"])
        return dict(rgba=s["rgba"], depth=s["depth"])
    if kind == "brick":
        return yoxel.render_volume(s["desc"], s["cams"], *s["size"], step_vox=s["step"],
                                   out=s["out"])
    if kind == "train":
        rgba = yoxel.volume_march(s["density"], s["albedo"], s["tv"], s["cams"], *s["size"])
        gd, ga = torch.autograd.grad(rgba, (s["density"], s["albedo"]), s["grad"])
        return dict(rgba=rgba, grad_density=gd, grad_albedo=ga)
    if kind == "batch":
        s["batch"].render()
        return s["out"]
    if kind == "svolive":
        s["renderer"].SetSceneDense(s["field"], s["depth"], 0.0, s["rgb"])
        s["renderer"].render_async(**s["out"])
        return s["out"]
    s["volume"].rebuild_dense(s["density"], s["levels"], s["rgb"])
    return yoxel.render_volume_rgba8(s["volume"].desc(), s["cams"], *s["size"], out=s["out"])


# ---- what a pass cannot do without --------------------------------------------------------

def _svo_work(px, rays, depth, out_bytes):
    # per ray a descent of `depth` levels and about as many sibling moves and returns, 20
    # operations each; per pixel one 40-byte node and one 8-byte attribute (most pixels end in
    # a leaf of their own), and the outputs
    return px * (48 + out_bytes), rays * depth * 3 * 20


def _march_work(rays, levels, point_bytes, out_bytes):
    # about a third of a ray's half-voxel samples through the volume are taken, 100 operations
    # each; a fifth of the bricks are occupied, each point read once
    side = 8 * 4 ** levels
    return (0.2 * side ** 3 * point_bytes + rays * out_bytes), rays * side * 0.7 * 100


def work(case):
    kind = case["kind"]
    px = case.get("width", 0) * case.get("height", 0) * case.get("cams", 1)
    if kind in ("svo", "lod", "edit", "svolive"):
        b, f = _svo_work(px, px * (1.6 if case.get("shadows") else 1), case["depth"], 12)
        if kind == "svolive":
            # the field once; a surface of 4 G^2 voxels written as nodes and leaf records
            b += 4.0 * 8 ** case["depth"] + 4 * 4 ** case["depth"] * 32
    elif kind == "ssna":
        b, f = _svo_work(px, px, case["depth"], 8)
        f += px * 300
    elif kind == "brick":
        b, f = _march_work(px, case["levels"], {F16: 6, F32: 16}.get(case["precision"], 8), 16)
    elif kind == "train":
        b, f = _march_work(px, case["levels"], 32, 48)
        f *= 4
    elif kind == "batch":
        b = f = 0
        for sp in _batch_specs(case):
            n = (sp["res"] + sp["odd"]) * sp["res"]
            x, y = _svo_work(n, n, sp["depth"], 4) if sp["svo"] else \
                _march_work(n, sp["levels"], 8, 16)
            b, f = b + x, f + y
    else:
        b, f = _march_work(px, case["levels"], 16, 4)
        b += 7.0 * (8 * 4 ** case["levels"] + 1) ** 3
    return dict(bytes=b, flops=f)


# ---- the same in 64 bits, by plain torch --------------------------------------------------

def _rays(cam, width, height):
    """Unnormalised pixel rays of a pinhole camera (forward component 1), (h*w, 3)."""
    pos, view, up, fov = cam

    def unit(v):
        return v / v.norm()
    f = unit(torch.tensor(view, dtype=torch.float64))
    right = unit(torch.linalg.cross(f, torch.tensor(up, dtype=torch.float64)))
    top = torch.linalg.cross(right, f)
    s = 2.0 * math.tan(math.radians(fov) / 2) / width
    x = (torch.arange(width, dtype=torch.float64) - width / 2) * s
    y = (torch.arange(height, dtype=torch.float64) - height / 2) * s
    u = f + right * x[None, :, None] - top * y[:, None, None]
    return torch.tensor(pos, dtype=torch.float64).cuda(), u.reshape(-1, 3).cuda()


def _directions(u):
    d = u / u.norm(dim=1, keepdim=True)
    return torch.where(d.abs() < 1e-5, torch.copysign(torch.full_like(d, 1e-5), d), d)


def _clip(o, d):
    a, b = (0.0 - o) / d, (1.0 - o) / d
    t0 = torch.minimum(a, b).amax(1).clamp_min(0.0)
    t1 = torch.maximum(a, b).amin(1)
    return t0, t1


def _first_solid(solid, o, d):
    """Distance at which each ray enters its first solid voxel, 0 where it meets none."""
    G = solid.shape[0]
    flat = solid.reshape(-1)
    t, t1 = _clip(o, d)
    out = torch.zeros_like(t)
    idx = (t < t1).nonzero()[:, 0]
    d, t = d[idx], t[idx]
    cell = ((o + d * t[:, None]) * G).floor().clamp_(0, G - 1).long()
    step = torch.where(d > 0, 1, -1)
    delta = (1.0 / (G * d)).abs()
    plane = ((cell + (step > 0)).double() / G - o) / d
    best, live = torch.zeros_like(t), torch.ones_like(t, dtype=torch.bool)
    for k in range(3 * G + 3):
        hit = flat[(cell[:, 2] * G + cell[:, 1]) * G + cell[:, 0]] & live
        best = torch.where(hit, t, best)
        t, e = plane.min(1)
        e = torch.nn.functional.one_hot(e, 3)
        cell = cell + step * e
        plane = plane + delta * e
        live = live & ~hit & ((cell >= 0) & (cell < G)).all(1)
        cell = cell.clamp(0, G - 1)
        if k % 32 == 31:  # the rays that ended leave
            out[idx] = best
            idx, cell, t, plane, step, delta, best = (v[live] for v in (idx, cell, t, plane, step,
                                                                        delta, best))
            live = torch.ones_like(idx, dtype=torch.bool)
            if idx.numel() == 0:
                break
    out[idx] = best
    return out


def _hit_t(case, seed):
    o, u = _rays(_camera(seed), case["width"], case["height"])
    solid = _field(case, seed) > 0
    return _first_solid(solid, o, _directions(u)), u


class _Dense:
    """A lattice and its occupied bricks, in 64 bits, as a pool of the given format stores it."""

    def __init__(self, levels, seed, half, shape=None):
        d, rgb = _lattice(levels, seed, shape)
        self.levels, self.nb = levels, 4 ** levels
        n = d.shape[0]
        self.n = n
        o = torch.nn.functional.max_pool3d(d[None, None].abs(), 9, 8)[0, 0] > 0
        self.occupied = o
        self.density = (d.half().double() if half else d.double()).reshape(-1)
        self.color = (rgb.reshape(-1, 3).double() if half
                      else rgb.reshape(-1, 3).float().mul(1.0 / 255.0).double() * 255.0)

    def march(self, o, d, step, visit=None):
        """(C, A) of each ray; visit(sample corners, weights, alpha, sigma, colour, T, C after)."""
        S = 8 * self.nb
        dt = float(torch.tensor(step / S, dtype=torch.float32))
        t0, t1 = _clip(o, d)
        R = d.shape[0]
        C, A = torch.zeros((R, 3), device="cuda", dtype=torch.float64), t0 * 0
        k0 = (t0 / dt).ceil()
        idx = (t0 < t1).nonzero()[:, 0]
        d, t0, t1, k0 = d[idx], t0[idx], t1[idx], k0[idx]
        c, a = C[idx], A[idx]
        off = torch.tensor([(j >> 2) * self.n * self.n + ((j >> 1) & 1) * self.n + (j & 1)
                            for j in range(8)], device="cuda")
        for k in range(int(math.sqrt(3) / dt) + 3):
            t = (k0 + k) * dt
            p = (o + d * t[:, None]) * S
            i = p.floor().clamp_(0, S - 1).long()
            f = (p - i).clamp_(0.0, 1.0)
            g = 1.0 - f
            occ = self.occupied[i[:, 2] >> 3, i[:, 1] >> 3, i[:, 0] >> 3] & (t < t1)
            q = (i[:, 2] * self.n + i[:, 1]) * self.n + i[:, 0]
            q = q[:, None] + off
            w = torch.stack([(f if j & 1 else g)[:, 0] * (f if j & 2 else g)[:, 1] *
                             (f if j & 4 else g)[:, 2] for j in range(8)], 1)
            sig = (self.density[q] * w).sum(1) * occ
            col = (self.color[q] * w[:, :, None]).sum(1) / 255.0
            al = sig.clamp(0.0, 1.0)
            T = 1.0 - a
            c = c + (T * al)[:, None] * col
            a = a + T * al
            if visit is not None:
                visit(idx, q, w, occ, sig, al, col, T, c, a)
            if k % 8 == 7:
                C[idx], A[idx] = c, a
                live = (a <= 0.99) & (t < t1)
                idx, d, t1, k0, c, a = (v[live] for v in (idx, d, t1, k0, c, a))
                if idx.numel() == 0:
                    break
            else:
                over = a > 0.99
                t1 = torch.where(over, torch.full_like(t1, -1.0), t1)
        C[idx], A[idx] = c, a
        return torch.cat([C, A[:, None]], 1)


def _exact_rgba(vol, cams, width, height, step):
    return torch.stack([vol.march(o, _directions(u), step).reshape(height, width, 4)
                        for o, u in (_rays(c, width, height) for c in cams)])


def _exact_train(case, seed):
    w, h = case["width"], case["height"]
    vol = _Dense(case["levels"], seed, False, FITTED)
    g = torch.randn((case["cams"], h, w, 4), generator=_gen(seed + 3), device="cuda").double()
    grad = torch.zeros((vol.n ** 3, 4), device="cuda", dtype=torch.float64)
    frames = []
    for k, cam in enumerate(_cameras(case, seed)):
        o, u = _rays(cam, w, h)
        d = _directions(u)
        out = vol.march(o, d, 0.5)
        frames.append(out.reshape(h, w, 4))
        gk = g[k].reshape(-1, 4)
        total = (gk * out).sum(1)

        def visit(idx, q, wt, occ, sig, al, col, T, c, a):
            gr = gk[idx]
            gc = (gr[:, :3] * col).sum(1) + gr[:, 3]
            after = (gr[:, :3] * c).sum(1) + gr[:, 3] * a
            om = 1.0 - al
            dal = T * gc - torch.where(om > 0, (total[idx] - after) / om.clamp_min(1e-300), 0.0)
            # saturate' = 1 on [0, 1): empty points still receive gradient
            ds = torch.where((sig < 1.0) & occ & (T >= 0.01), dal, 0.0)
            wa = T * al
            rows = torch.cat([gr[:, None, :3] * (wa[:, None] * wt)[:, :, None],
                              (ds[:, None] * wt)[:, :, None]], 2)
            grad.index_add_(0, q.reshape(-1), rows.reshape(-1, 4))
        vol.march(o, d, 0.5, visit)
    # into the pool's layout: bricks breadth-first (4-ary digits, x lowest); a far-side point
    # holds its owner's gradient, 0 where its owner does not exist
    z, y, x = vol.occupied.nonzero(as_tuple=True)
    key = torch.zeros_like(x)
    for lev in range(vol.levels):
        sh = 2 * (vol.levels - 1 - lev)
        key = key * 64 + (((x >> sh) & 3) | (((y >> sh) & 3) << 2) | (((z >> sh) & 3) << 4))
    order = key.argsort()
    x, y, z = x[order], y[order], z[order]
    p = torch.arange(729, device="cuda")
    lx, ly, lz = 8 * x[:, None] + p % 9, 8 * y[:, None] + (p // 9) % 9, 8 * z[:, None] + p // 81
    own = torch.nn.functional.pad(vol.occupied, (0, 1, 0, 1, 0, 1))[lz >> 3, ly >> 3, lx >> 3]
    v = grad[(lz * vol.n + ly) * vol.n + lx] * own[:, :, None]
    return dict(rgba=torch.stack(frames), grad_density=v[:, :, 3].contiguous(),
                grad_albedo=v[:, :, :3].contiguous())


def _exact_ssna(case, seed):
    """View depth blurred in passes whose reach shrinks with distance."""
    w, h = case["width"], case["height"]
    t, u = _hit_t(case, seed)
    far, voxel = 1e30, 1.0 / 2048.0
    thr, pad = 4.0 / 2048.0, 0.3 * 4.0 / 2048.0
    z = torch.where(t > 0, t / u.norm(dim=1), far).reshape(h, w)
    hit = (t > 0).reshape(h, w)
    pix = math.radians(FOV) / w
    ky = {o: math.exp(-float(o * o)) for o in range(-2, 3)}
    for i in range(5):
        limit = 5.0 * voxel / (pix * 3.0 * (i + 1))
        zp = torch.nn.functional.pad(z[None], (2, 2, 2, 2), value=-1.0)[0]
        acc, tot = torch.zeros_like(z), torch.zeros_like(z)
        for oy in range(-2, 3):
            for ox in range(-2, 3):
                s = zp[2 + oy:2 + oy + h, 2 + ox:2 + ox + w]
                m = zp[2 - oy:2 - oy + h, 2 - ox:2 - ox + w]
                inside, minside = s >= 0, m >= 0
                near = z > s + thr
                ok = inside & (~near | (minside & ~(z > m + thr)))
                v = torch.where(near, torch.where(m > z + thr, z + pad, m),
                                torch.where(s > z + thr, z + pad, s))
                k = ky[ox] * ky[oy] * ok
                acc += torch.where(ok, v, torch.zeros_like(v)) * k
                tot += k
        z = torch.where((z > 0) & (z <= limit), acc / tot, z)
    return dict(rgba=None, depth=torch.where(hit, z, 0.0))


def exact(case, seed):
    kind = case["kind"]
    if kind in ("svo", "svolive", "edit"):
        t, _ = _hit_t(case, seed)
        return dict(rgba=None, hit=None, hit_t=t.reshape(case["height"], case["width"]))
    if kind == "ssna":
        return _exact_ssna(case, seed)
    if kind == "brick":
        vol = _Dense(case["levels"], seed, case["precision"] != F32)
        return _exact_rgba(vol, _cameras(case, seed), case["width"], case["height"], case["step"])
    if kind == "train":
        if case["cams"] * case["width"] * case["height"] > 1500000:
            return None  # half a minute
        return _exact_train(case, seed)
    if kind == "batch":
        got = []
        for i, sp in enumerate(_batch_specs(case)):
            if sp["svo"]:
                got.append(None)
            else:
                vol = _Dense(sp["levels"], seed + i, True)
                got.append(_exact_rgba(vol, [_camera(seed + i)], sp["res"] + sp["odd"],
                                       sp["res"], 0.5)[0])
        return got
    return None  # a cut-off ray's distance and 8-bit colours have no such value
