"""The workloads by which this framework's speed is judged: what its users ask of it.

A user traces a 2-D scene of mirrors and glass into light segments, accumulates the segments
into an image and resolves the image.  They do so one frame at a time (a still scene rendered
again and again, an edited scene uploaded every frame, a large final frame), stage by stage,
with segments of their own, as a batch of scenes and as a stream of requests.  Every case goes
through the package's public entry points (``Context``, ``Tracer``, the C ABI of ``lg.h``).

The scenes are seeded: the seed decides every shape, position, colour and light.  Images come
back whole: RGBA16F as a float16 tensor, the fixed-point accumulation as int64, the F32
accumulation as float32, the export as bytes.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from light_garden_gb300 import abi, workloads as W
from light_garden_gb300.runtime import Context
from light_garden_gb300.scene import (Circle, Material, Object, PointLight, Rect, SpotLight, pack)
from light_garden_gb300.tracer import Tracer


def listed():
    return [
        # the smallest frame: one light, a glass disc and a mirror, rendered over and over by a
        # preview (the repository's plain configuration: 4096 rays, 512x512, FP32 accumulation)
        {"name": "preview", "kind": "preview", "rays": 4096, "bounces": 8, "width": 512, "height": 512, "accum": "f32"},
        # the editor: the scene changes, so every frame packs, uploads, traces and downloads
        # (a window of odd size, a handful of objects and lights)
        {"name": "editor", "kind": "editor", "rays": 6000, "lights": 2, "objects": 12, "bounces": 5, "width": 1021,
         "height": 683},
        # every shape of the scene model, stage by stage (trace, accumulate), then the 8-bit
        # export that a screenshot takes
        {"name": "shapes_export", "kind": "shapes", "rays": 1 << 14, "objects": 48, "bounces": 12, "width": 1024,
         "height": 768},
        # a scene of 64 plain objects in full HD, exact: the repository's mid configuration
        {"name": "mid_frame", "kind": "mid", "rays": 1 << 18, "lights": 8, "objects": 64, "bounces": 16, "width": 1920,
         "height": 1080, "precision": "exact", "accum": "fixed"},
        # the same kind of frame as a quick look: double-float trace, FP32 accumulation
        {"name": "mid_draft", "kind": "mid", "rays": 1 << 15, "lights": 8, "objects": 64, "bounces": 16, "width": 1279,
         "height": 719, "precision": "fast", "accum": "f32"},
        # the headline: constructive geometry, deep reflections, a large canvas and a string-mod
        # overlay, exact (the benchmark's frame at three sixteenths of its rays)
        {"name": "csg_frame", "kind": "csg", "rays": 3 << 18, "objects": 256, "bounces": 32, "width": 4096,
         "height": 4096, "precision": "exact"},
        # the same geometry in double-float at a size that one accumulation pass takes
        {"name": "csg_fast", "kind": "csg", "rays": 1 << 17, "objects": 200, "bounces": 24, "width": 2048,
         "height": 2048, "precision": "fast"},
        # segments that another tracer left on the device, drawn without allocating
        {"name": "segments_device", "kind": "segments_device", "count": 400_000, "mean_px": 90.0, "width": 1600,
         "height": 1200, "accum": "fixed", "blend": "add"},
        # segments in host memory, drawn into an FP32 image of odd size
        {"name": "segments_host", "kind": "segments_host", "count": 150_001, "mean_px": 60.0, "width": 1277,
         "height": 717, "accum": "f32", "blend": "add"},
        # nested string art: the crossings of the outer mod's lines are found at upload
        {"name": "string_art", "kind": "string", "outer": 1200, "width": 1024, "height": 1024},
        # many scenes of mixed sizes in one call, at a sixteenth of their rays
        {"name": "batch", "kind": "batch", "scenes": 64, "scale": 1.0 / 16},
        # the render server: requests of mixed sizes submitted together, stepped until all are
        # done, every image polled
        {"name": "serve", "kind": "serve", "scenes": 24, "scale": 1.0 / 32},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the ranges above: every kind, sizes over their whole range."""
    kind = rng.choice(["preview", "editor", "shapes", "mid", "mid", "csg", "csg", "segments_device", "segments_host",
                       "string", "batch", "serve"])
    if kind == "preview":
        return {"kind": kind, "rays": _log(rng, 256, 1 << 16), "bounces": rng.randint(2, 20),
                "width": _log(rng, 128, 1024), "height": _log(rng, 128, 1024), "accum": rng.choice(["f32", "fixed"])}
    if kind == "editor":
        return {"kind": kind, "rays": _log(rng, 500, 12000), "lights": rng.randint(1, 4), "objects": rng.randint(1, 24),
                "bounces": rng.randint(2, 8), "width": _log(rng, 320, 1920), "height": _log(rng, 240, 1080)}
    if kind == "shapes":
        return {"kind": kind, "rays": _log(rng, 1 << 9, 1 << 15), "objects": _log(rng, 6, 96),
                "bounces": rng.randint(3, 16), "width": _log(rng, 256, 2048), "height": _log(rng, 256, 1536)}
    if kind == "mid":
        return {"kind": kind, "rays": _log(rng, 1 << 9, 1 << 18), "lights": rng.randint(1, 8),
                "objects": _log(rng, 8, 400), "bounces": rng.randint(4, 16), "width": _log(rng, 320, 2560),
                "height": _log(rng, 240, 1440), "precision": rng.choice(["exact", "exact", "fast"]),
                "accum": rng.choice(["fixed", "f32"])}
    if kind == "csg":
        return {"kind": kind, "rays": _log(rng, 1 << 12, 1 << 19), "objects": _log(rng, 12, 320),
                "bounces": rng.randint(4, 32), "width": _log(rng, 512, 4096), "height": _log(rng, 512, 4096),
                "precision": rng.choice(["exact", "exact", "fast"])}
    if kind in ("segments_device", "segments_host"):
        return {"kind": kind, "count": _log(rng, 100, 400_000), "mean_px": rng.uniform(8.0, 150.0),
                "width": _log(rng, 64, 2048), "height": _log(rng, 64, 2048), "accum": rng.choice(["fixed", "f32"]),
                "blend": rng.choice(["add", "add", "max"])}
    if kind == "string":
        return {"kind": kind, "outer": _log(rng, 64, 3000), "width": _log(rng, 256, 2048),
                "height": _log(rng, 256, 2048)}
    return {"kind": kind, "scenes": _log(rng, 2, 64 if kind == "batch" else 32),
            "scale": 1.0 / rng.choice([16, 32, 64, 128])}


# ---- scenes -----------------------------------------------------------------------------------
_ACCUM = {"f32": abi.LG_ACCUM_F32, "fixed": abi.LG_ACCUM_FIXED64}
_PRECISION = {"exact": abi.LG_PRECISION_EXACT, "fast": abi.LG_PRECISION_FAST}


def _canvas(p, case):
    p.width, p.height = case["width"], case["height"]
    p.max_bounce = case["bounces"]
    return p


def _preview(case, seed):
    """The plain configuration's scene, its parts moved a little by the seed."""
    r = np.random.default_rng(seed)
    w = W.plain_small(accum=_ACCUM[case["accum"]], num_rays=case["rays"])
    w.objects[0] = Object(abi.LG_OBJ_CIRCLE, Circle((float(r.uniform(-0.1, 0.1)), float(r.uniform(-0.1, 0.1))),
                                                    float(r.uniform(0.15, 0.3))), Material(1.5))
    w.lights[0].position = (float(r.uniform(-0.9, -0.7)), float(r.uniform(-0.2, 0.2)))
    _canvas(w.params, case)
    return w


def _editor(case, seed):
    """What a user puts together by hand: discs, boxes, lenses and flat mirrors, point and spot lights."""
    r = np.random.default_rng(seed)
    objects, lights = [], []
    for k in range(case["objects"]):
        c = (float(r.uniform(-1.2, 1.2)), float(r.uniform(-0.8, 0.8)))
        size, a = float(r.uniform(0.05, 0.2)), float(r.uniform(0, 2 * math.pi))
        what = k % 4
        if what == 0:
            objects.append(Object(abi.LG_OBJ_CIRCLE, Circle(c, size), Material(float(r.uniform(1.2, 1.7)))))
        elif what == 1:
            objects.append(Object(abi.LG_OBJ_RECT, Rect(c, 2 * size, size, (math.cos(a), math.sin(a))),
                                  Material(float(r.uniform(1.2, 1.7)))))
        elif what == 2:
            objects.append(Object.new_mirror(c, (c[0] + size * math.cos(a), c[1] + size * math.sin(a))))
        else:
            objects.append(Object.new_lens(c, 2 * size, 2.5 * size))
    for k in range(case["lights"]):
        pos = (float(r.uniform(-1.2, 1.2)), float(r.uniform(-0.8, 0.8)))
        color = tuple(float(v) for v in r.uniform(0.2, 1.0, 3)) + (1.0,)
        if k % 2 == 0:
            lights.append(PointLight(pos, case["rays"], color))
        else:
            a = float(r.uniform(0, 2 * math.pi))
            lights.append(SpotLight(pos, float(r.uniform(0.3, 1.2)), (math.cos(a), math.sin(a)), case["rays"], color))
    return objects, lights


def _frame(case, seed):
    kind = case["kind"]
    if kind == "preview":
        w = _preview(case, seed)
    elif kind == "shapes":
        w = W.shapes_scene(seed=seed, rays_per_light=case["rays"], n_objects=case["objects"])
        _canvas(w.params, case)
    elif kind == "mid":
        w = W.mid_scene(seed=seed, accum=_ACCUM[case["accum"]], rays_per_light=case["rays"],
                        n_objects=case["objects"], n_lights=case["lights"])
        _canvas(w.params, case).precision = _PRECISION[case["precision"]]
    elif kind == "csg":
        w = W.csg_scene(seed=seed, total_rays=case["rays"], n_objects=case["objects"], width=case["width"],
                        height=case["height"])
        _canvas(w.params, case).precision = _PRECISION[case["precision"]]
    else:
        w = W.nested_string_mod_art(curve=seed % 4, width=case["width"], height=case["height"],
                                    outer_modulo=case["outer"])
        w.params.string_mod.num += seed % 13
        w.params.string_mod.turns = 1
    return w


def _segments(case, seed):
    """Segments as a trace leaves them: starts spread over the canvas, every direction, lengths of
    an exponential spread, colours faded by a few bounces (x0, y0, x1, y1, r, g, b, a per row)."""
    n, w, h = case["count"], case["width"], case["height"]
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    u = torch.rand((n, 8), generator=g, device="cuda", dtype=torch.float32)
    x, y = (2.0 * u[:, 0] - 1.0) * (w / h), 2.0 * u[:, 1] - 1.0
    a = 2.0 * math.pi * u[:, 2]
    length = -torch.log1p(-u[:, 3]) * (2.0 * case["mean_px"] / h)
    fade = torch.pow(0.5, 6.0 * u[:, 4])
    out = torch.stack([x, y, x + length * torch.cos(a), y + length * torch.sin(a), fade * u[:, 5], fade * u[:, 6],
                       fade * u[:, 7], torch.ones_like(x)], dim=1)
    return out.contiguous()


def _segment_params(case):
    p = abi.params_default()
    p.width, p.height, p.accum = case["width"], case["height"], _ACCUM[case["accum"]]
    if case["blend"] == "max":
        p.color_blend = abi.lg_blend_component(abi.LG_BF_ONE, abi.LG_BF_ONE, abi.LG_BO_MAX)
        p.alpha_blend = abi.lg_blend_component(abi.LG_BF_ONE, abi.LG_BF_ONE, abi.LG_BO_MAX)
    return p


def _scenes(case, seed):
    """Scenes of the mixed generator; their canvases go round its four sizes."""
    ws = W.batch_scenes(seed=seed, count=case["scenes"])
    for k, w in enumerate(ws):
        w.params.width = w.params.height = (256, 512, 1024, 2048)[k % 4]
    return [W.scale_rays(w, case["scale"]).packed() for w in ws]


# ---- the cases --------------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind == "editor":
        t = Tracer(case["width"], case["height"])
        t.max_bounce = case["bounces"]
        t.objects, t.lights = _editor(case, seed)
        return {"kind": kind, "tracer": t}
    if kind == "segments_device":
        dtype = torch.int64 if case["accum"] == "fixed" else torch.float32
        return {"kind": kind, "lib": abi.load(), "params": _segment_params(case), "segments": _segments(case, seed),
                "image": torch.empty((case["height"], case["width"], 4), dtype=dtype, device="cuda")}
    ctx = Context(device=0)
    if kind == "segments_host":
        segs = _segments(case, seed).cpu().numpy().view(abi.segment_dtype()).reshape(-1)
        ctx.upload(pack([], [], _segment_params(case)))
        return {"kind": kind, "ctx": ctx, "segments": segs}
    if kind == "batch":
        scenes = _scenes(case, seed)
        ctx.batch_upload(scenes)
        out = torch.empty((ctx.batch_pixels(), 4), dtype=torch.float16, device="cuda")
        return {"kind": kind, "ctx": ctx, "image": out}
    if kind == "serve":
        ctx.serve_begin(hbm_budget_bytes=12 << 30, max_slots=64)
        return {"kind": kind, "ctx": ctx, "scenes": _scenes(case, seed)}
    w = _frame(case, seed)
    pk = w.packed()
    out = torch.empty((pk.params.height, pk.params.width, 4), dtype=torch.float16, device="cuda")
    if kind != "string":  # string art is uploaded by every pass
        ctx.upload(pk)
    return {"kind": kind, "ctx": ctx, "scene": pk, "image": out}


def run(state):
    kind = state["kind"]
    if kind == "editor":
        return state["tracer"].render_to_texture().view(np.float16)
    if kind == "segments_device":
        segs, img = state["segments"], state["image"]
        st = state["lib"].lg_accumulate_segments_noalloc(
            C.c_void_p(segs.data_ptr()), segs.shape[0], C.byref(state["params"]), C.c_void_p(img.data_ptr()),
            C.c_void_p(torch.cuda.current_stream().cuda_stream), None)
        if st != abi.LG_OK:
            raise abi.LgError(st, "lg_accumulate_segments_noalloc")
        return img
    ctx = state["ctx"]
    if kind == "segments_host":
        ctx.accumulate_segments(state["segments"])
        return ctx.accum()
    if kind == "shapes":
        ctx.trace()
        ctx.accumulate()
        return {"export": ctx.resolve_rgba8(), "accumulation": ctx.accum()}
    if kind == "batch":
        img = state["image"]
        ctx.batch_render_into(img.data_ptr(), img.numel() * 2, True)
        return img
    if kind == "serve":
        ids = [ctx.serve_submit(sc) for sc in state["scenes"]]
        images = {}
        while len(images) < len(ids):
            if ctx.serve_step()["finished"]:
                for i in ids:
                    if i not in images:
                        img = ctx.serve_poll(i)
                        if img is not None:
                            images[i] = img.view(np.float16)
        return [images[i] for i in ids]
    img = state["image"]
    if kind == "string":
        ctx.upload(state["scene"])
    ctx.render_into(img.data_ptr(), img.stride(0) * img.element_size(), True)
    return img


# Ray visits per primary ray, about (it depends on the scene): every bounce off glass splits a ray
# in two until its colour falls below the cutoff.
_VISITS = {"preview": 2.0, "editor": 4.0, "shapes": 40.0, "mid": 60.0, "csg": 360.0}
_FLOPS_PER_VISIT = 150.0  # the FP64 solve of one hit, Snell, Fresnel and the two child directions
_FLOPS_PER_PIXEL = 6.0    # the raster rule and four channel sums of one drawn pixel


def work(case):
    """One pass: every primary followed to its end, every segment pixel summed, the image written."""
    kind = case["kind"]
    if kind in ("segments_device", "segments_host"):
        n, px = case["count"], case["width"] * case["height"]
        per = 4 * (8 if case["accum"] == "fixed" else 4)
        return {"bytes": 32.0 * n + per * px, "flops": _FLOPS_PER_PIXEL * n * 0.8 * case["mean_px"]}
    if kind == "string":
        px = case["width"] * case["height"]
        m = case["outer"]
        return {"bytes": 8.0 * px + 32.0 * m, "flops": 20.0 * m * (m - 1) + _FLOPS_PER_PIXEL * 6000 * 0.3 * case["width"]}
    if kind in ("batch", "serve"):
        # the mean scene of the generator: 180 k rays, 73 visits a ray, 1.4 M pixels, 37 pixels a segment
        rays = 180_000.0 * case["scale"] * case["scenes"]
        return {"bytes": 8.0 * 1.4e6 * case["scenes"], "flops": rays * 73 * (_FLOPS_PER_VISIT + 37 * _FLOPS_PER_PIXEL)}
    rays = case["rays"] * {"preview": 1, "editor": case.get("lights", 1), "shapes": 4, "mid": case.get("lights", 1),
                           "csg": 1}[kind]
    full = {"preview": 8, "editor": 5, "shapes": 12, "mid": 16, "csg": 32}[kind]
    visits = rays * max(1.0, _VISITS[kind] * min(1.0, case["bounces"] / full))
    px = case["width"] * case["height"]
    per_segment = 0.15 * case["height"] * _FLOPS_PER_PIXEL
    out = 36.0 if kind == "shapes" else 8.0
    return {"bytes": out * px, "flops": visits * (_FLOPS_PER_VISIT + per_segment)}


# ---- 64-bit values ----------------------------------------------------------------------------
# The raster rule in double: pixel centres of the major axis in [ceil(a - 1/2), ceil(b - 1/2)),
# the minor pixel floor(v); vertex and sample coordinates are those of the f32 vertex format.
def _f32(x):
    return x.to(torch.float32).to(torch.float64)


def _raster64(segs, width, height, blend):
    """Sum (or maximum) of the segments' contributions over the clear colour, in float64."""
    dev = segs.device
    img = torch.zeros((height * width, 4), dtype=torch.float64, device=dev)
    img[:, 3] = 1.0
    s = segs.to(torch.float64)
    sc, cx = height * 0.5, width * 0.5
    X0, Y0, X1, Y1 = _f32(s[:, 0] * sc + cx), _f32(-s[:, 1] * sc + sc), _f32(s[:, 2] * sc + cx), _f32(-s[:, 3] * sc + sc)
    xm = _f32((X1 - X0).abs()) >= _f32((Y1 - Y0).abs())
    ua, va = torch.where(xm, X0, Y0), torch.where(xm, Y0, X0)
    ub, vb = torch.where(xm, X1, Y1), torch.where(xm, Y1, X1)
    sw = ub < ua
    ua, ub = torch.where(sw, ub, ua), torch.where(sw, ua, ub)
    va, vb = torch.where(sw, vb, va), torch.where(sw, va, vb)
    du = _f32(ub - ua)
    ok = du > 0
    slope = _f32(_f32(vb - va) / torch.where(ok, du, torch.ones_like(du)))
    nmaj = torch.where(xm, float(width), float(height)).to(torch.float64)
    lo = torch.ceil(_f32(ua - 0.5)).clamp(min=0.0)
    hi = torch.minimum(torch.ceil(_f32(ub - 0.5)), nmaj)
    cnt = torch.where(ok, (hi - lo).clamp(min=0.0), torch.zeros_like(lo)).to(torch.int64)
    col = s[:, 4:8].clone()
    if blend == "add":
        col[:, 3] = col[:, 3] * col[:, 3]
    step = 1 << 17
    for b in range(0, s.shape[0], step):
        e = slice(b, min(s.shape[0], b + step))
        c = cnt[e]
        if int(c.sum()) == 0:
            continue
        k = torch.repeat_interleave(torch.arange(c.shape[0], device=dev), c) + b
        start = torch.cumsum(c, 0) - c
        i = lo[k] + (torch.arange(k.shape[0], device=dev) - start[k - b]).to(torch.float64)
        j = torch.floor(_f32(_f32(_f32(i + 0.5) - ua[k]) * slope[k] + va[k]))
        x, y = torch.where(xm[k], i, j), torch.where(xm[k], j, i)
        on = (x >= 0) & (x < width) & (y >= 0) & (y < height)
        px = (y[on] * width + x[on]).to(torch.int64)
        if blend == "add":
            img.index_add_(0, px, col[k[on]])
        else:
            img.scatter_reduce_(0, px[:, None].expand(-1, 4), col[k[on]], "amax")
    return img.reshape(height, width, 4)


def _hits(obj, o, d):
    """All hits of one object of the editor or the preview: (t, normal x, normal y) columns, inf where none."""
    def circle(c, r):
        f = o - torch.tensor(c, dtype=torch.float64, device=o.device)
        b, q = (f * d).sum(1), (f * f).sum(1) - r * r
        disc = b * b - q
        sq = torch.sqrt(disc.clamp(min=0.0))
        out = []
        for t in (-b - sq, -b + sq):
            t = torch.where((disc >= 0) & (t > 1e-9), t, torch.full_like(t, math.inf))
            n = (f + d * torch.where(t < math.inf, t, torch.zeros_like(t))[:, None]) / r
            out.append((t, n[:, 0], n[:, 1]))
        return out
    g = obj.geo
    inf = torch.full((o.shape[0],), math.inf, dtype=torch.float64, device=o.device)
    if isinstance(g, Circle):
        return circle(g.origin, g.radius)
    if isinstance(g, Rect):
        c, s = g.rotation
        f = o - torch.tensor(g.origin, dtype=torch.float64, device=o.device)
        lo = [c * f[:, 0] + s * f[:, 1], -s * f[:, 0] + c * f[:, 1]]
        ld = [c * d[:, 0] + s * d[:, 1], -s * d[:, 0] + c * d[:, 1]]
        h = (0.5 * g.width, 0.5 * g.height)
        out = []
        for ax in (0, 1):
            for sg in (-1.0, 1.0):
                t = (sg * h[ax] - lo[ax]) / ld[ax]
                ok = (t > 1e-9) & ((lo[1 - ax] + t * ld[1 - ax]).abs() <= h[1 - ax])
                n = (c * sg, s * sg) if ax == 0 else (-s * sg, c * sg)
                out.append((torch.where(ok, t, inf), torch.full_like(t, n[0]), torch.full_like(t, n[1])))
        return out
    if obj.kind == abi.LG_OBJ_LENS:
        cs = [(g.origin[0] + k.origin[0], g.origin[1] + k.origin[1], k.radius) for k in (g.a, g.b)]
        out = []
        for me, other in ((cs[0], cs[1]), (cs[1], cs[0])):
            for t, nx, ny in circle(me[:2], me[2]):
                p = o + d * torch.where(t < math.inf, t, torch.zeros_like(t))[:, None]
                inside = (p[:, 0] - other[0]) ** 2 + (p[:, 1] - other[1]) ** 2 <= other[2] ** 2
                out.append((torch.where(inside, t, inf), nx, ny))
        return out
    e = (g.b[0] - g.a[0], g.b[1] - g.a[1])
    den = d[:, 0] * e[1] - d[:, 1] * e[0]
    wx, wy = g.a[0] - o[:, 0], g.a[1] - o[:, 1]
    t, u = (wx * e[1] - wy * e[0]) / den, (wx * d[:, 1] - wy * d[:, 0]) / den
    le = math.hypot(*e)
    ok = (u >= 0) & (u <= 1) & (t > 1e-9)
    return [(torch.where(ok, t, inf), torch.full_like(t, -e[1] / le), torch.full_like(t, e[0] / le))]


def _inside(obj, p):
    g = obj.geo
    if isinstance(g, Circle):
        return (p[:, 0] - g.origin[0]) ** 2 + (p[:, 1] - g.origin[1]) ** 2 <= g.radius ** 2
    if isinstance(g, Rect):
        c, s = g.rotation
        x, y = p[:, 0] - g.origin[0], p[:, 1] - g.origin[1]
        return ((c * x + s * y).abs() <= 0.5 * g.width) & ((-s * x + c * y).abs() <= 0.5 * g.height)
    if obj.kind == abi.LG_OBJ_LENS:
        r = torch.ones(p.shape[0], dtype=torch.bool, device=p.device)
        for k in (g.a, g.b):
            r &= (p[:, 0] - g.origin[0] - k.origin[0]) ** 2 + (p[:, 1] - g.origin[1] - k.origin[1]) ** 2 <= k.radius ** 2
        return r
    return torch.zeros(p.shape[0], dtype=torch.bool, device=p.device)


def _trace64(objects, lights, bounces, aspect):
    """The segments of a scene of discs, boxes, lenses and flat mirrors, followed in float64."""
    dev = torch.device("cuda")
    O, D, K, N = [], [], [], []
    for l in lights:
        i = torch.arange(l.num_rays, dtype=torch.float64, device=dev)
        if isinstance(l, PointLight):
            a = i * (2.0 * math.pi) / l.num_rays
        else:
            a = math.atan2(l.spot_direction[1], l.spot_direction[0]) - 0.5 * l.spot_angle + (i + 1) / l.num_rays * l.spot_angle
        O.append(torch.tensor(l.position, dtype=torch.float64, device=dev).expand(l.num_rays, 2))
        D.append(torch.stack([torch.cos(a), torch.sin(a)], 1))
        K.append(torch.tensor(l.color, dtype=torch.float64, device=dev).expand(l.num_rays, 4))
        n = 1.0
        for ob in objects:  # the last object that holds the light
            if ob.material_opt and bool(_inside(ob, torch.tensor([l.position], dtype=torch.float64, device=dev))[0]):
                n = ob.material_opt.refractive_index
        N.append(torch.full((l.num_rays,), n, dtype=torch.float64, device=dev))
    o, d, k, n1 = torch.cat(O), torch.cat(D), torch.cat(K), torch.cat(N)
    segs = []
    for _ in range(bounces):
        if o.shape[0] == 0:
            break
        live = ~((k[:, :3] < 0.001).all(1) | (k[:, 3] < 0.001))
        o, d, k, n1 = o[live], d[live], k[live], n1[live]
        m = o.shape[0]
        t = torch.full((m,), math.inf, dtype=torch.float64, device=dev)
        nx, ny = torch.zeros_like(t), torch.zeros_like(t)
        hit = torch.full((m,), -1, dtype=torch.int64, device=dev)
        for q, ob in enumerate(objects):
            for ht, hx, hy in _hits(ob, o, d):
                near = ht < t
                t, nx, ny = torch.where(near, ht, t), torch.where(near, hx, nx), torch.where(near, hy, ny)
                hit = torch.where(near, q, hit)
        out = hit < 0
        tx = torch.where(d[:, 0] > 0, aspect - o[:, 0], -aspect - o[:, 0]) / d[:, 0]
        ty = torch.where(d[:, 1] > 0, 1.0 - o[:, 1], -1.0 - o[:, 1]) / d[:, 1]
        t = torch.where(out, torch.minimum(tx, ty), t)
        p = o + d * t[:, None]
        draw_it = ~out | ((o[:, 0].abs() <= aspect) & (o[:, 1].abs() <= 1.0))
        segs.append(torch.cat([o, p, k], 1)[draw_it])
        h = ~out
        oh, dh, kh, nh, ph = o[h], d[h], k[h], n1[h], p[h]
        nv, hh = torch.stack([nx, ny], 1)[h], hit[h]
        glass = torch.tensor([ob.material_opt is not None for ob in objects], device=dev)[hh]
        index = torch.tensor([ob.material_opt.refractive_index if ob.material_opt else 1.0 for ob in objects],
                             dtype=torch.float64, device=dev)
        mid = 0.5 * (oh + ph)
        from_in = torch.zeros(oh.shape[0], dtype=torch.bool, device=dev)
        other = torch.ones(oh.shape[0], dtype=torch.float64, device=dev)
        for q in reversed(range(len(objects))):  # the first other object that holds the point
            if objects[q].material_opt:
                from_in |= (hh == q) & _inside(objects[q], mid)
                other = torch.where((hh != q) & _inside(objects[q], ph), index[q], other)
        n2 = torch.where(from_in, other, index[hh])
        ci = -(dh * nv).sum(1)
        nv = torch.where((ci < 0)[:, None], -nv, nv)
        ci = ci.abs()
        refl = dh + nv * (2.0 * ci)[:, None]
        eta = nh / n2
        kk = 1.0 - eta * eta * (1.0 - ci * ci)
        ct = torch.sqrt(kk.clamp(min=0.0))
        refr = dh * eta[:, None] + nv * (eta * ci - ct)[:, None]
        rs, rp = (nh * ci - n2 * ct) / (nh * ci + n2 * ct), (nh * ct - n2 * ci) / (nh * ct + n2 * ci)
        R = torch.where(glass & (kk >= 0), 0.5 * (rs * rs + rp * rp), torch.ones_like(ci))
        ones = torch.ones_like(R)
        go = glass & (kk >= 0)
        c1 = kh * torch.stack([R, R, R, ones], 1)
        c2 = (kh * torch.stack([1 - R, 1 - R, 1 - R, ones], 1))[go]
        o, d, k, n1 = torch.cat([ph, ph[go]]), torch.cat([refl, refr[go]]), torch.cat([c1, c2]), torch.cat([nh, n2[go]])
    return torch.cat(segs) if segs else torch.zeros((0, 8), dtype=torch.float64, device=dev)


def _half(img):
    return img.to(torch.float32).to(torch.float16).to(torch.float64)


def exact(case, seed):
    """The preview's and the editor's image and the F32 accumulation of given segments, in 64 bits.
    A whole deep frame, a batch and a server's images would take minutes."""
    kind = case["kind"]
    if kind in ("segments_device", "segments_host") and case["accum"] == "f32":
        return _raster64(_segments(case, seed), case["width"], case["height"], case["blend"])
    if kind in ("preview", "editor"):
        if kind == "preview":
            w = _preview(case, seed)
            objects, lights = w.objects, w.lights
        else:
            objects, lights = _editor(case, seed)
        aspect = float(np.float32(case["width"]) / np.float32(case["height"]))
        segs = _trace64(objects, lights, case["bounces"], aspect)
        return _half(_raster64(segs.to(torch.float32), case["width"], case["height"], "add"))
    return None
