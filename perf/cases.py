"""Performance cases of the framework: ray queries, rendering, serving,
denoising and the denoiser's training, each through the public entry points.

`listed()` names the cases, `draw(rng)` gives one more of the same ranges,
`prepare(case, seed)` makes what a program holds before the call, `run(state)`
is one pass, `work(case)` the bytes and operations that pass cannot do
without, and `exact(case, seed)` its result in 64 bits, where that is a
computed number (Monte Carlo images have none).

Scenes, servers and contexts are made once and shared by the states, as a
program loads its scene once; seeds change the rays, the sample ranges, the
requests, the images and the weights.
"""
import functools
import math

import numpy as np
import torch

from cudaraytracer_b200 import Context, Scene, Svgf, scenes
from cudaraytracer_b200.kpcn import Kpcn, conv3x3_backward_data, conv3x3_backward_weights, conv3x3_forward
from cudaraytracer_b200.serve import RenderRequest, Server

DEVICE = "cuda:0"
FIELD_SPHERES = 64  # the 1.31M-triangle field of the benchmark: 64 level-5 icospheres
FIELD_LEVEL = 5


# --------------------------------------------------------------------------
# cases
# --------------------------------------------------------------------------


def listed():
    return [
        # a picking or probe query: a thousand closest hits in a small scene, bound by the call itself
        {"name": "query_box_1k", "kind": "closest", "scene": "box", "spheres": 0, "level": 0, "n": 1000},
        # a light-baking batch in the Cornell box: closest hits, then visibility
        {"name": "trace_box_1m", "kind": "trace", "scene": "box", "spheres": 0, "level": 0, "n": 1 << 20},
        # an ordinary batch in a scene of 82k triangles, of odd size
        {"name": "trace_mid_200k", "kind": "trace", "scene": "field", "spheres": 16, "level": 4, "n": 200003},
        # the benchmark's headline: 16M closest hits and 16M visibility queries in 1.31M triangles
        {"name": "trace_field_16m", "kind": "trace", "scene": "field", "spheres": FIELD_SPHERES,
         "level": FIELD_LEVEL, "n": 1 << 24},
        # an interactive preview: a small frame at a few samples per pixel
        {"name": "frame_box_256", "kind": "frame", "scene": "box", "width": 256, "height": 256, "spp": 4},
        # one progressive sample of a full-HD frame: four materials, sky and sun, 16 bounces
        {"name": "frame_field_1080p", "kind": "frame", "scene": "field", "width": 1920, "height": 1080, "spp": 1},
        # a batch of training views
        {"name": "views_box_16", "kind": "views", "views": 16, "width": 256, "height": 256, "spp": 8},
        # a burst of render requests over resident scenes, images read back to the host
        {"name": "serve_box_8", "kind": "serve", "requests": 8, "width": 256, "height": 256, "spp": 16},
        # one denoised full-HD frame of a moving camera, history in place
        {"name": "svgf_1080p", "kind": "svgf", "width": 1920, "height": 1080},
        # the learned denoiser on a full-HD frame
        {"name": "kpcn_1080p", "kind": "kpcn", "n": 1, "height": 1080, "width": 1920},
        # the gradients of one training batch of the learned denoiser
        {"name": "kpcn_grad_8x128", "kind": "grad", "n": 8, "height": 128, "width": 128},
        # forward and both gradients of one convolution layer at half resolution
        {"name": "conv_64_540p", "kind": "conv", "n": 1, "height": 540, "width": 960, "cin": 64, "cout": 64},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["closest", "trace", "trace", "frame", "frame", "views", "serve", "svgf", "kpcn", "grad", "conv",
                       "conv"])
    if kind in ("closest", "trace"):
        c = {"kind": kind, "scene": rng.choice(["box", "field"]), "spheres": 0, "level": 0}
        if c["scene"] == "field":
            c["spheres"], c["level"] = rng.choice([(1, 3), (4, 3), (16, 4), (16, 5), (64, 5)])
        c["n"] = _log_int(rng, 500, 100_000 if kind == "closest" else 1 << 23) | 1
        return c
    if kind == "frame":
        scene = rng.choice(["box", "field"])
        w, h = _log_int(rng, 96, 1920), _log_int(rng, 64, 1080)
        return {"kind": kind, "scene": scene, "width": w, "height": h,
                "spp": max(1, min(_log_int(rng, 1, 16), (1 << 21) // (w * h)))}
    if kind == "views":
        w, h, v = _log_int(rng, 64, 512), _log_int(rng, 64, 512), rng.randint(2, 24)
        return {"kind": kind, "views": v, "width": w, "height": h,
                "spp": max(1, min(rng.randint(1, 16), (1 << 23) // (w * h * v)))}
    if kind == "serve":
        w, h, r = _log_int(rng, 64, 512), _log_int(rng, 64, 512), rng.randint(2, 16)
        return {"kind": kind, "requests": r, "width": w, "height": h,
                "spp": max(1, min(rng.randint(1, 16), (1 << 23) // (w * h * r)))}
    if kind == "svgf":
        return {"kind": kind, "width": _log_int(rng, 200, 1920), "height": _log_int(rng, 120, 1080)}
    if kind == "kpcn":
        w, h = 4 * _log_int(rng, 16, 480), 4 * _log_int(rng, 16, 270)
        return {"kind": kind, "n": max(1, min(rng.randint(1, 8), 2073600 // (w * h))), "height": h, "width": w}
    if kind == "grad":
        return {"kind": kind, "n": rng.randint(1, 8), "height": 4 * _log_int(rng, 8, 48),
                "width": 4 * _log_int(rng, 8, 48)}
    w, h = _log_int(rng, 33, 1920), _log_int(rng, 33, 1080)
    return {"kind": "conv", "n": max(1, min(rng.randint(1, 8), 518400 // (w * h))), "height": h, "width": w,
            "cin": rng.choice([16, 32, 48, 64, 96, 128, 160]), "cout": rng.choice([16, 32, 48, 64, 80, 96, 128])}


# --------------------------------------------------------------------------
# what a program loads once
# --------------------------------------------------------------------------


@functools.lru_cache(maxsize=None)
def _context():
    return Context(0)


@functools.lru_cache(maxsize=None)
def _triangles(scene, spheres, level):
    if scene == "box":
        return scenes.cornell_box().triangles()
    return scenes.icosphere_field(n_spheres=spheres, level=level, with_env=False).triangles()


@functools.lru_cache(maxsize=None)
def _query_scene(scene, spheres, level):
    tris = _triangles(scene, spheres, level)
    return Scene.from_triangles(_context(), tris), torch.from_numpy(tris).to(DEVICE).view(-1, 3, 3)


@functools.lru_cache(maxsize=8)
def _render_scene(scene, width, height, variant=0):
    if scene == "box":
        spec = scenes.cornell_box(width=width, height=height, max_bounces=12, seed=variant or None)
    else:
        spec = _field_spec()
        spec.camera = dict(spec.camera, resolution=[width, height])
    return Scene.from_spec(_context(), spec)


@functools.lru_cache(maxsize=None)
def _field_spec():
    return scenes.icosphere_field(n_spheres=FIELD_SPHERES, level=FIELD_LEVEL)


def _gen(seed):
    return torch.Generator(device=DEVICE).manual_seed(int(seed))


# --------------------------------------------------------------------------
# ray queries
# --------------------------------------------------------------------------


def _unit(g, n):
    z = torch.rand(n, generator=g, device=DEVICE) * 2 - 1
    phi = torch.rand(n, generator=g, device=DEVICE) * (2 * math.pi)
    r = torch.sqrt(torch.clamp(1 - z * z, min=0))
    return torch.stack([r * torch.cos(phi), r * torch.sin(phi), z], 1)


def _random_rays(tris, n, g):
    """Origins uniform in the scene's box, directions uniform on the sphere."""
    lo, hi = tris.reshape(-1, 3).amin(0), tris.reshape(-1, 3).amax(0)
    out = torch.empty((n, 8), device=DEVICE)
    out[:, 0:3] = lo + (hi - lo) * torch.rand((n, 3), generator=g, device=DEVICE)
    out[:, 3] = 0.0
    out[:, 4:7] = _unit(g, n)
    out[:, 7] = 1e8
    return out


def _random_queries(tris, n, g):
    """Shading points uniform in the scene's box, light points uniform on random triangles."""
    lo, hi = tris.reshape(-1, 3).amin(0), tris.reshape(-1, 3).amax(0)
    out = torch.empty((n, 12), device=DEVICE)
    out[:, 0:3] = lo + (hi - lo) * torch.rand((n, 3), generator=g, device=DEVICE)
    out[:, 3:6] = _unit(g, n)
    t = tris[torch.randint(0, tris.shape[0], (n,), generator=g, device=DEVICE)]
    u = torch.rand((n, 2), generator=g, device=DEVICE)
    u = torch.where(u.sum(1, keepdim=True) > 1, 1 - u, u)
    e1, e2 = t[:, 1] - t[:, 0], t[:, 2] - t[:, 0]
    out[:, 6:9] = t[:, 0] + u[:, 0:1] * e1 + u[:, 1:2] * e2
    out[:, 9:12] = torch.nn.functional.normalize(torch.linalg.cross(e1, e2), dim=1, eps=1e-30)
    return out


def _prepare_trace(case, seed):
    scene, tris = _query_scene(case["scene"], case["spheres"], case["level"])
    g = _gen(seed)
    n = case["n"]
    s = {"kind": case["kind"], "scene": scene, "rays": _random_rays(tris, n, g),
         "hits": torch.empty((n, 4), device=DEVICE)}
    if case["kind"] == "trace":
        s["queries"] = _random_queries(tris, n, g)
        s["occluded"] = torch.empty((n,), dtype=torch.uint8, device=DEVICE)
    return s


def _run_trace(s):
    hits = s["scene"].trace_closest(s["rays"], s["hits"])
    out = {"t": hits[:, 0], "prim": hits.view(torch.int32)[:, 1], "bary": hits[:, 2:4]}
    if s["kind"] == "trace":
        out["occluded"] = s["scene"].trace_shadow(s["queries"], s["occluded"])
    return out


def _exact_trace(case, seed):
    """Every triangle against every ray; only where that is little work."""
    if case["scene"] != "box":
        return None
    s = _prepare_trace(case, seed)
    tris = _query_scene("box", 0, 0)[1].double()
    v0, e1, e2 = tris[:, 0], tris[:, 1] - tris[:, 0], tris[:, 2] - tris[:, 0]
    n = case["n"]
    t_out = torch.full((n,), 1e8, dtype=torch.float64, device=DEVICE)
    b_out = torch.zeros((n, 2), dtype=torch.float64, device=DEVICE)
    o, d = s["rays"][:, 0:3].double(), s["rays"][:, 4:7].double()
    for k in range(tris.shape[0]):
        s1 = torch.linalg.cross(d, e2[k].expand_as(d))
        sv = o - v0[k]
        s2 = torch.linalg.cross(sv, e1[k].expand_as(sv))
        det = (s1 * e1[k]).sum(1)
        inv = 1.0 / torch.where(det > 0, det, torch.ones_like(det))
        t, b1, b2 = (s2 * e2[k]).sum(1) * inv, (s1 * sv).sum(1) * inv, (s2 * d).sum(1) * inv
        ok = (det > 0) & (b1 >= 0) & (b2 >= 0) & (b1 + b2 <= 1) & (t >= 0) & (t < t_out)
        t_out = torch.where(ok, t, t_out)
        b_out = torch.where(ok[:, None], torch.stack([b1, b2], 1), b_out)
    out = {"t": t_out, "prim": None, "bary": b_out}
    if case["kind"] == "trace":
        out["occluded"] = None
    return out


# --------------------------------------------------------------------------
# rendering
# --------------------------------------------------------------------------


def _first_sample(seed):
    return (int(seed) * 7919 % (1 << 20)) * 64


def _prepare_frame(case, seed):
    h, w = case["height"], case["width"]
    return {"scene": _render_scene(case["scene"], w, h), "spp": case["spp"], "first": _first_sample(seed),
            "direct": torch.empty((h, w, 4), device=DEVICE), "indirect": torch.empty((h, w, 4), device=DEVICE)}


def _run_frame(s):
    s["direct"].zero_()
    s["indirect"].zero_()
    s["scene"].render_device(s["direct"], s["indirect"], s["spp"], first_sample=s["first"])
    return {"direct": s["direct"], "indirect": s["indirect"]}


def _orbit(scene, n, seed):
    """Poses around the open side of the box."""
    rng = np.random.default_rng(int(seed))
    c = scene.camera()
    return [{"target": list(c["target"]), "distance": float(c["distance"]) * float(rng.uniform(0.85, 1.1)),
             "theta_deg": float(rng.uniform(75, 105)), "phi_deg": float(rng.uniform(-20, 20)),
             "fovy_deg": float(c["fovy_deg"])} for _ in range(n)]


def _prepare_views(case, seed):
    n, h, w = case["views"], case["height"], case["width"]
    scene = _render_scene("box", w, h)
    return {"scene": scene, "spp": case["spp"], "cameras": _orbit(scene, n, seed), "first": _first_sample(seed),
            "direct": torch.empty((n, h, w, 4), device=DEVICE), "indirect": torch.empty((n, h, w, 4), device=DEVICE)}


def _run_views(s):
    s["direct"].zero_()
    s["indirect"].zero_()
    s["scene"].render_views(s["cameras"], s["direct"], s["indirect"], s["spp"], first_sample=s["first"])
    return {"direct": s["direct"], "indirect": s["indirect"]}


@functools.lru_cache(maxsize=None)
def _server():
    srv = Server(_context(), paths_per_pass=4 << 20)
    resident = [Scene.from_spec(_context(), scenes.cornell_box(max_bounces=12, seed=100 + k)) for k in range(4)]
    for sc in resident:
        srv.add_scene(sc)
    return srv, resident


def _prepare_serve(case, seed):
    srv, resident = _server()
    reqs = []
    for k in range(case["requests"]):
        sid = k % len(resident)
        reqs.append(RenderRequest(sid, case["width"], case["height"], case["spp"],
                                  _orbit(resident[sid], 1, int(seed) * 1000 + k)[0], seed=int(seed) * 1000 + k))
    return {"server": srv, "requests": reqs}


def _run_serve(s):
    srv = s["server"]
    ids = [srv.submit(r) for r in s["requests"]]
    srv.drain()
    out = []
    for rid, r in zip(ids, s["requests"]):
        out.append(srv.result(rid, r.width, r.height))
        srv.release(rid)
    return out


# --------------------------------------------------------------------------
# SVGF
# --------------------------------------------------------------------------

SVGF_FRAMES = 6  # frames of the orbit before the timed one: the history is in place


def _svgf_inputs(case, seed):
    """Frames of a camera orbiting the field by 0.5 degrees a frame: 1-sample images and G-buffers."""
    w, h = case["width"], case["height"]
    scene = _render_scene("field", w, h)
    cam = dict(scene.camera())
    first, frames, prev = _first_sample(seed), [], None
    for f in range(SVGF_FRAMES + 1):
        phi = cam["phi_deg"] + 0.5 * f
        scene.set_camera_orbit(cam["target"], cam["distance"], cam["theta_deg"], phi, cam["fovy_deg"])
        d, i = torch.zeros((h, w, 4), device=DEVICE), torch.zeros((h, w, 4), device=DEVICE)
        scene.render_device(d, i, 1, first_sample=first + f)
        frames.append((d, i, scene.gbuffer(prev_camera=prev)))
        prev = scene.camera()
    scene.set_camera_orbit(cam["target"], cam["distance"], cam["theta_deg"], cam["phi_deg"], cam["fovy_deg"])
    return frames


def _prepare_svgf(case, seed):
    w, h = case["width"], case["height"]
    frames = _svgf_inputs(case, seed)
    sv = Svgf(_context(), w, h)
    out_d, out_i = torch.empty((h, w, 4), device=DEVICE), torch.empty((h, w, 4), device=DEVICE)
    for f in range(SVGF_FRAMES):
        d, i, g = frames[f]
        sv.frame(g, frames[f - 1][2] if f else g, d, i, out_d, out_i)
    return {"svgf": sv, "cur": frames[-1], "prev": frames[-2], "out_d": out_d, "out_i": out_i}


def _run_svgf(s):
    d, i, g = s["cur"]
    s["svgf"].frame(g, s["prev"][2], d, i, s["out_d"], s["out_i"])
    return {"direct": s["out_d"], "indirect": s["out_i"]}


def _lum(c):
    return 0.2126 * c[..., 0] + 0.7152 * c[..., 1] + 0.0722 * c[..., 2]


def _tap(x, dy, dx):
    """x[(y + dy), (x + dx)] with the coordinates clamped, and where they lie inside."""
    h, w = x.shape[:2]
    ys = torch.arange(h, device=x.device) + dy
    xs = torch.arange(w, device=x.device) + dx
    return x[ys.clamp(0, h - 1)][:, xs.clamp(0, w - 1)]


def _inside(h, w, dy, dx):
    ys = torch.arange(h, device=DEVICE)[:, None] + dy
    xs = torch.arange(w, device=DEVICE)[None, :] + dx
    return (ys >= 0) & (ys < h) & (xs >= 0) & (xs < w)


def _decode_gbuffer(g):
    nm = g["normal_mat"].int() & 0xFFFF
    bm = g["bary_mesh"].int() & 0xFFFF
    n = nm[..., :3].double() / 65535.0 * 2 - 1
    n = n / n.norm(dim=-1, keepdim=True)
    md = g["motion_depth"].double()
    return {"n": n, "mat": nm[..., 3], "mesh": bm[..., 3], "tri": g["pos_tri"][..., 3].int(), "mx": md[..., 0],
            "my": md[..., 1], "z": md[..., 2], "dz": md[..., 3]}


def _exact_temporal(cur, last, hist, cd, ci):
    """The temporal pass: colours with variance, moments and history lengths."""
    h, w = cur["z"].shape
    y, x = torch.meshgrid(torch.arange(h, device=DEVICE), torch.arange(w, device=DEVICE), indexing="ij")
    mvx, mvy = cur["mx"] * w * 0.5, cur["my"] * h * 0.5
    dist = (mvx * mvx + mvy * mvy).sqrt()
    px, py = x + 0.5 - mvx, y + 0.5 - mvy
    inside = (px >= 0.5) & (px < w - 0.5) & (py >= 0.5) & (py < h - 0.5)
    table = torch.cat([hist["d"], hist["i"], hist["md"], hist["mi"], hist["len"][..., None]], -1).reshape(h * w, -1)

    def tap(tx, ty):
        ok = (tx >= 0) & (tx < w) & (ty >= 0) & (ty < h)
        k = ty.clamp(0, h - 1) * w + tx.clamp(0, w - 1)
        at = lambda v: v.reshape((h * w,) + v.shape[2:])[k]  # noqa: E731
        zl = at(last["z"])
        thr = torch.maximum(cur["dz"], at(last["dz"])) * (dist + 1) + 0.1 * torch.maximum(cur["z"], zl)
        ok = ok & (cur["mesh"] == at(last["mesh"])) & (cur["mat"] == at(last["mat"])) & (cur["tri"] == at(last["tri"]))
        return ok & ((cur["n"] * at(last["n"])).sum(-1) >= 0.9) & ((cur["z"] - zl).abs() <= thr), k

    fx, fy = px - 0.5, py - 0.5
    bx, by = fx.floor().long(), fy.floor().long()
    frx, fry = fx - bx, fy - by
    every = torch.ones_like(inside)
    acc, tw = torch.zeros((h, w, table.shape[1]), dtype=torch.float64, device=DEVICE), torch.zeros_like(px)
    for oy in (0, 1):
        for ox in (0, 1):
            ok, k = tap(bx + ox, by + oy)
            wt = (frx if ox else 1 - frx) * (fry if oy else 1 - fry) * ok
            every, tw, acc = every & ok, tw + wt, acc + table[k] * wt[..., None]
    good = every & (tw > 1e-6)
    acc2, tw2 = torch.zeros_like(acc), torch.zeros_like(tw)
    cx, cy = px.floor().long().clamp(0, w - 1), py.floor().long().clamp(0, h - 1)
    for oy in (-1, 0, 1):
        for ox in (-1, 0, 1):
            ok, k = tap(cx + ox, cy + oy)
            wt = (0.25 if ox else 0.5) * (0.25 if oy else 0.5) * ok
            tw2, acc2 = tw2 + wt, acc2 + table[k] * wt[..., None]
    acc = torch.where(good[..., None], acc / tw.clamp(min=1e-12)[..., None], acc2 / tw2.clamp(min=1e-12)[..., None])
    valid = inside & (good | (tw2 > 1e-6))
    acc = acc * valid[..., None]
    length = torch.where(valid, ((acc[..., 10] + 0.5).floor().clamp(min=1) + 1).clamp(max=24), torch.ones_like(px))
    a = torch.where(valid, 1 / length, torch.ones_like(px))
    out = {"len": length}
    for key, c, o, m in (("d", cd, 0, 6), ("i", ci, 3, 8)):
        lum = _lum(c)
        out[key] = a[..., None] * c + (1 - a[..., None]) * acc[..., o:o + 3]
        out["m" + key] = torch.stack([a * lum + (1 - a) * acc[..., m], a * lum * lum + (1 - a) * acc[..., m + 1]], -1)
        var = out["m" + key][..., 1] - out["m" + key][..., 0] ** 2
        out["v" + key] = torch.where(valid, var, torch.ones_like(var))
    return out


def _exact_weights(cur, dy, dx, same, wz, sn, cl, nl, light):
    nn = (cur["n"] * _tap(cur["n"], dy, dx)).sum(-1).clamp(min=0)
    return same * nn ** sn * torch.exp(wz - (cl - nl).abs() * light)


def _exact_svgf(case, seed):
    """The reference's filter in 64 bits over the whole sequence: reprojection,
    7x7 variance where the history is short, five a-trous passes (only the
    last frame's, as they do not feed the history)."""
    h, w = case["height"], case["width"]
    hist = {"d": torch.zeros((h, w, 3), dtype=torch.float64, device=DEVICE)}
    hist.update(i=hist["d"], md=hist["d"][..., :2], mi=hist["d"][..., :2], len=hist["d"][..., 0])
    last = None
    for f, (d, i, g) in enumerate(_svgf_inputs(case, seed)):
        cur = _decode_gbuffer(g)
        cd, ci = d[..., :3].double(), i[..., :3].double()
        if f == 0:
            ld, li = _lum(cd), _lum(ci)
            hist = {"d": cd, "i": ci, "md": torch.stack([ld, ld * ld], -1), "mi": torch.stack([li, li * li], -1),
                    "len": torch.ones((h, w), dtype=torch.float64, device=DEVICE)}
        else:
            hist = _exact_temporal(cur, last, hist, cd, ci)
        last = cur
    ids = cur["mat"] | (cur["mesh"] << 16)
    dz = cur["dz"].clamp(min=1e-4)
    col, var = {"d": hist["d"], "i": hist["i"]}, {"d": hist["vd"], "i": hist["vi"]}
    lum = {k: _lum(col[k]) for k in "di"}
    acc = {k: torch.zeros((h, w, 6), dtype=torch.float64, device=DEVICE) for k in "di"}
    for dy in range(-3, 4):
        for dx in range(-3, 4):
            same = (_inside(h, w, dy, dx) & (ids == _tap(ids, dy, dx))).double()
            wz = -(cur["z"] - _tap(cur["z"], dy, dx)).abs() / (dz * math.hypot(dx, dy) + 1e-4)
            for k in "di":
                nl = _tap(lum[k], dy, dx)
                light = (torch.maximum(lum[k], nl).clamp(min=1e-4) if k == "d" else lum[k]).sqrt() / 8.0
                wt = _exact_weights(cur, dy, dx, same, wz, 256.0, lum[k], nl, light)[..., None]
                m = _tap(hist["m" + k], dy, dx)
                acc[k] += wt * torch.cat([_tap(col[k], dy, dx), m, torch.ones_like(m[..., :1])], -1)
    short = hist["len"] < 4
    for k in "di":
        f = acc[k][..., :5] / acc[k][..., 5:].clamp(min=1e-6)
        v = (f[..., 4] - f[..., 3] ** 2).clamp(min=0) * 4 / hist["len"]
        col[k] = torch.where(short[..., None], f[..., :3], col[k])
        var[k] = torch.where(short, v, var[k])
    n_hist = hist["len"]
    boot = ((4 - n_hist) / 3).clamp(0, 1)
    for p in range(5):
        step, kern = 1 << p, (0.375, 0.25, 0.0625)
        new_c, new_v = {}, {}
        lum = {k: _lum(col[k]) for k in "di"}
        sd = {}
        for k in "di":
            fv, fw = torch.zeros_like(boot), torch.zeros_like(boot)
            for dy in (-1, 0, 1):
                for dx in (-1, 0, 1):
                    wt = (0.25 if dx else 0.5) * (0.25 if dy else 0.5) * _inside(h, w, dy, dx)
                    fv, fw = fv + wt * _tap(var[k], dy, dx).clamp(min=0), fw + wt
            sd[k] = (fv / fw.clamp(min=1e-6)).sqrt() + 1e-3
            new_c[k] = torch.zeros((h, w, 3), dtype=torch.float64, device=DEVICE)
            new_v[k] = [torch.zeros_like(boot), torch.zeros_like(boot)]
        sz = dz * (1 + 2.5 * boot)
        sl = {"d": 8 * (1 + 2 * boot), "i": 8 * (1 + 1.5 * boot)}
        sn = (256 * (1 - 0.85 * boot)).clamp(min=8)
        for dy in range(-2, 3):
            for dx in range(-2, 3):
                ty, tx = dy * step, dx * step
                same = (_inside(h, w, ty, tx) & (ids == _tap(ids, ty, tx))).double()
                wz = -(cur["z"] - _tap(cur["z"], ty, tx)).abs() / (sz * (math.hypot(dx, dy) * step) + 1e-6)
                hc = torch.where(boot > 0, 0.5 + 0.5 * (_tap(n_hist, ty, tx) / 4).clamp(max=1), torch.ones_like(boot))
                for k in "di":
                    nl = _tap(lum[k], ty, tx)
                    ref = torch.maximum(lum[k], nl) if k == "d" else lum[k]
                    light = ref.clamp(min=1e-4).sqrt() / (sl[k] * sd[k])
                    wt = _exact_weights(cur, ty, tx, same, wz, sn, lum[k], nl, light)
                    wt = wt * hc * (kern[abs(dx)] * kern[abs(dy)])
                    new_c[k] += wt[..., None] * _tap(col[k], ty, tx)
                    new_v[k][0] += wt
                    new_v[k][1] += wt * wt * _tap(var[k], ty, tx).clamp(min=0)
        for k in "di":
            tw = new_v[k][0]
            some = tw > 1e-6
            col[k] = torch.where(some[..., None], new_c[k] / tw.clamp(min=1e-6)[..., None], col[k])
            var[k] = torch.where(some, new_v[k][1] / tw.clamp(min=1e-6) ** 2, torch.ones_like(tw))
    return {"direct": torch.cat([col["d"], var["d"][..., None]], -1),
            "indirect": torch.cat([col["i"], var["i"][..., None]], -1)}


# --------------------------------------------------------------------------
# the learned denoiser
# --------------------------------------------------------------------------


def _weights(seed):
    """Weights of a network with He-scaled layers and a filter that is not uniform."""
    rng = np.random.default_rng(int(seed))
    parts = []
    for k, (cin, cout) in enumerate(Kpcn.SPEC):
        real_in, real_out = (13 if k == 0 else cin), (25 if k == len(Kpcn.SPEC) - 1 else cout)
        w = np.zeros((9, cout, cin), np.float32)
        std = math.sqrt(2.0 / (9 * real_in)) if k < len(Kpcn.SPEC) - 1 else 0.05
        w[:, :real_out, :real_in] = rng.normal(size=(9, real_out, real_in)) * std
        b = np.zeros(cout, np.float32)
        b[:real_out] = rng.normal(size=real_out) * 0.05
        parts += [w.ravel(), b]
    return np.concatenate(parts)


def _images(case, seed):
    """Feature planes, noisy radiance and a target with the value ranges of a
    rendered view: smooth surfaces, a few materials, heavy-tailed noise."""
    n, h, w = case["n"], case["height"], case["width"]
    g = _gen(seed)
    smooth = torch.randn((n, 9, max(2, h // 16), max(2, w // 16)), generator=g, device=DEVICE)
    smooth = torch.nn.functional.interpolate(smooth, size=(h, w), mode="bilinear", align_corners=False)
    smooth = smooth.permute(0, 2, 3, 1)
    target = torch.zeros((n, h, w, 4), device=DEVICE)
    target[..., :3] = torch.exp(0.8 * smooth[..., :3] - 1.0)
    noisy = torch.zeros((n, h, w, 4), device=DEVICE)
    gain = torch.randn((n, h, w, 3), generator=g, device=DEVICE)
    noisy[..., :3] = target[..., :3] * torch.exp(0.7 * gain - 0.25)
    feat = torch.zeros((n, h, w, 16), device=DEVICE)
    feat[..., 0:3] = torch.log1p(noisy[..., :3])
    feat[..., 3:6] = torch.sigmoid(2 * smooth[..., 3:6]).mul(4).round().div(4)
    feat[..., 6:9] = torch.nn.functional.normalize(smooth[..., 6:9], dim=-1)
    feat[..., 9] = 0.5 + 0.1 * smooth[..., 0]
    feat[..., 12] = 0.5
    return feat.to(torch.bfloat16).contiguous(), noisy, target


def _prepare_kpcn(case, seed):
    net = Kpcn(_context(), seed=1)
    net.set_params(_weights(seed))
    feat, noisy, target = _images(case, seed)
    return {"net": net, "feat": feat, "noisy": noisy, "target": target, "out": torch.empty_like(noisy)}


def _run_kpcn(s):
    return s["net"].forward(s["feat"], s["noisy"], s["out"])


def _run_grad(s):
    loss = s["net"].train_step(s["feat"], s["noisy"], s["target"], 0.0)
    return {"loss": loss, "grads": s["net"].get_grads()}


def _conv64(x, w):
    """3x3 convolution of (n, h, w, c) by (9, cout, cin) as nine matrix products."""
    n, h, wd, c = x.shape
    p = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1))
    out = None
    for t in range(9):
        y = p[:, t // 3:t // 3 + h, t % 3:t % 3 + wd].reshape(-1, c) @ w[t].T
        out = y if out is None else out + y
    return out.view(n, h, wd, -1)


def _forward64(params, feat):
    layers, off = [], 0
    for cin, cout in Kpcn.SPEC:
        w = params[off:off + 9 * cin * cout].view(9, cout, cin)
        layers.append((w, params[off + 9 * cin * cout:off + 9 * cin * cout + cout]))
        off += 9 * cin * cout + cout
    relu = torch.relu
    conv = lambda k, x: _conv64(x, layers[k][0]) + layers[k][1]  # noqa: E731
    pool = lambda x: (x[:, 0::2, 0::2] + x[:, 0::2, 1::2] + x[:, 1::2, 0::2] + x[:, 1::2, 1::2]) * 0.25  # noqa: E731
    up = lambda x: x.repeat_interleave(2, 1).repeat_interleave(2, 2)  # noqa: E731
    e0 = relu(conv(1, relu(conv(0, feat))))
    e1 = relu(conv(3, relu(conv(2, pool(e0)))))
    e2 = relu(conv(5, relu(conv(4, pool(e1)))))
    d1 = relu(conv(7, relu(conv(6, torch.cat([up(e2), e1], -1)))))
    d0 = relu(conv(9, relu(conv(8, torch.cat([up(d1), e0], -1)))))
    return conv(10, d0)[..., :25]


def _filter64(logits, noisy):
    n, h, w, _ = logits.shape
    wt = torch.softmax(logits, -1)
    ys, xs = torch.arange(h, device=DEVICE), torch.arange(w, device=DEVICE)
    out = torch.zeros((n, h, w, 3), dtype=torch.float64, device=DEVICE)
    for k in range(25):
        v = noisy[:, (ys + k // 5 - 2).clamp(0, h - 1)][:, :, (xs + k % 5 - 2).clamp(0, w - 1)]
        out = out + wt[..., k:k + 1] * v[..., :3]
    return out


def _exact_kpcn(case, seed):
    feat, noisy, _ = _images(case, seed)
    params = torch.from_numpy(_weights(seed)).to(DEVICE).double()
    with torch.no_grad():
        out = _filter64(_forward64(params, feat.double()), noisy.double())
    return torch.nn.functional.pad(out, (0, 1))


def _exact_grad(case, seed):
    feat, noisy, target = _images(case, seed)
    params = torch.from_numpy(_weights(seed)).to(DEVICE).double().requires_grad_()
    out = _filter64(_forward64(params, feat.double()), noisy.double())
    ref = target[..., :3].double()
    loss = ((out - ref) ** 2 / (ref ** 2 + 0.01)).mean()
    loss.backward()
    return {"loss": loss.item(), "grads": params.grad}


def _prepare_conv(case, seed):
    n, h, w, ci, co = (case[k] for k in ("n", "height", "width", "cin", "cout"))
    g = _gen(seed)
    x = torch.relu(torch.randn((n, h, w, ci), generator=g, device=DEVICE)).to(torch.bfloat16)  # a ReLU output
    wt = (torch.randn((9, co, ci), generator=g, device=DEVICE) * math.sqrt(2.0 / (9 * ci))).to(torch.bfloat16)
    return {"x": x, "w": wt, "wt": wt.transpose(1, 2).contiguous(),
            "bias": torch.randn((co,), generator=g, device=DEVICE) * 0.05,
            "g": (torch.randn((n, h, w, co), generator=g, device=DEVICE) * 1e-3).to(torch.bfloat16),
            "y": torch.empty((n, h, w, co), dtype=torch.bfloat16, device=DEVICE),
            "dx": torch.empty((n, h, w, ci), dtype=torch.bfloat16, device=DEVICE),
            "dw": torch.empty((9, co, ci), device=DEVICE)}


def _run_conv(s):
    ctx = _context()
    s["dw"].zero_()
    return {"y": conv3x3_forward(ctx, s["x"], s["w"], s["bias"], relu=True, out=s["y"]),
            "dx": conv3x3_backward_data(ctx, s["g"], s["wt"], mask=s["x"], out=s["dx"]),
            "dw": conv3x3_backward_weights(ctx, s["x"], s["g"], dw=s["dw"])}


def _exact_conv(case, seed):
    s = _prepare_conv(case, seed)
    x, w, g = s["x"].double(), s["w"].double(), s["g"].double()
    n, h, wd, ci = x.shape
    p = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1))
    gf = g.reshape(-1, g.shape[-1])
    dw = [gf.T @ p[:, t // 3:t // 3 + h, t % 3:t % 3 + wd].reshape(-1, ci) for t in range(9)]
    dx = _conv64(g, w.flip(0).transpose(1, 2))
    return {"y": torch.relu(_conv64(x, w) + s["bias"].double()), "dx": dx * (x > 0), "dw": torch.stack(dw)}


# --------------------------------------------------------------------------
# entry points
# --------------------------------------------------------------------------

_KINDS = {
    "closest": (_prepare_trace, _run_trace, _exact_trace),
    "trace": (_prepare_trace, _run_trace, _exact_trace),
    "frame": (_prepare_frame, _run_frame, None),
    "views": (_prepare_views, _run_views, None),
    "serve": (_prepare_serve, _run_serve, None),
    "svgf": (_prepare_svgf, _run_svgf, _exact_svgf),
    "kpcn": (_prepare_kpcn, _run_kpcn, _exact_kpcn),
    "grad": (_prepare_kpcn, _run_grad, _exact_grad),
    "conv": (_prepare_conv, _run_conv, _exact_conv),
}


def prepare(case, seed):
    return case["kind"], _KINDS[case["kind"]][0](case, seed)


def run(state):
    kind, s = state
    return _KINDS[kind][1](s)


def exact(case, seed):
    fn = _KINDS[case["kind"]][2]
    return fn(case, seed) if fn else None


def work(case):
    k = case["kind"]
    if k in ("closest", "trace"):
        # rays and queries in, hits and flags out; a ray tests at least one box (24 operations)
        n = case["n"]
        return {"bytes": 48.0 * n + (49.0 * n if k == "trace" else 0), "flops": 24.0 * n * (2 if k == "trace" else 1)}
    if k in ("frame", "views", "serve"):
        # the two accumulators of every pixel written; a camera ray and a box test per sample
        px = case["width"] * case["height"] * case.get("views", case.get("requests", 1))
        return {"bytes": 32.0 * px, "flops": 64.0 * px * case["spp"]}
    if k == "svgf":
        # two noisy images, two G-buffers, the history read and written, two images out
        px = case["width"] * case["height"]
        return {"bytes": px * (32.0 + 2 * 48 + 2 * 52 + 32), "flops": px * 5 * 25 * 40.0}
    px = case["n"] * case["height"] * case["width"]
    if k in ("kpcn", "grad"):
        scale = [1, 1, 4, 4, 16, 16, 4, 4, 1, 1, 1]
        fl = sum(18.0 * ci * co / s for (ci, co), s in zip(Kpcn.SPEC, scale)) * px
        params = sum(9 * ci * co + co for ci, co in Kpcn.SPEC)
        if k == "kpcn":
            return {"bytes": px * (32.0 + 16 + 16) + 2.0 * params, "flops": fl}
        return {"bytes": px * (32.0 + 16 + 16) + 4.0 * params, "flops": 3 * fl}
    ci, co = case["cin"], case["cout"]
    # forward reads x and writes y, the data gradient reads g and x and writes dx, the weight gradient reads x and g
    return {"bytes": px * 2.0 * (ci + co + co + ci + ci + ci + co) + 9.0 * ci * co * (2 + 2 + 4),
            "flops": 3 * 18.0 * ci * co * px}
