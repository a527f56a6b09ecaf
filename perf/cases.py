"""The work that a program using this framework has it do, as cases that can be timed.

Every case goes through a public entry point: the `processing` mirror (Pipeline, Render,
EntityBuffer, Canvas), the batch renderer, or the serving calls of the C ABI. The ranges:

  frame     one pass and the image read back (Pipeline.render, Pipeline.get_image): what a viewer
            does again and again while the camera rests
  passes    several samples per pixel in one call (Render.render_passes): offline frames
  example   the same over the scene types of the hy and eu examples, which the generic
            kernels serve (Render.render_passes)
  batch     many views of both geometries, sizes and object counts in one launch sequence
  serve     a burst of interactive and batch requests through the server, images read back

Sizes are those of the repository's workloads (scene.config0-2, batch.config3,
serve.make_requests, the bench's example scenes) and ragged ones between them; scenes, cameras
and pixel seeds come from the seed.
"""
import ctypes
import math

import numpy as np
import torch

from hypertrace_b200 import _lib
from hypertrace_b200 import batch as B
from hypertrace_b200 import processing as P
from hypertrace_b200 import scene as S
from hypertrace_b200 import serve as V
from hypertrace_b200 import types as T

GAMMA = 1.0 / 2.2


def listed():
    return [
        # the smallest call: one pass of a small Euclidean view, where latency counts
        dict(name="frame-eu-320x240", kind="frame", geometry="eu", width=320, height=240, objects=9, hops=4,
             address_width=32, double_support=False, flags=0),
        # a viewer's pass over the ordinary hyperbolic view
        dict(name="frame-hy-800x600", kind="frame", geometry="hy", width=800, height=600, objects=18, hops=6,
             address_width=32, double_support=False, flags=0),
        # a viewer's pass over the large hyperbolic view
        dict(name="frame-hy-1080p", kind="frame", geometry="hy", width=1920, height=1080, objects=200, hops=8,
             address_width=32, double_support=False, flags=0),
        # an offline Euclidean frame of an odd size, serialized on a 64-bit host
        dict(name="passes-eu-1917x1077", kind="passes", geometry="eu", width=1917, height=1077, objects=25, hops=5,
             passes=16, address_width=64, double_support=False, flags=0),
        # the ordinary offline frame
        dict(name="passes-hy-800x600", kind="passes", geometry="hy", width=800, height=600, objects=18, hops=6,
             passes=64, address_width=32, double_support=False, flags=0),
        # the headline frame
        dict(name="passes-hy-1080p", kind="passes", geometry="hy", width=1920, height=1080, objects=200, hops=8,
             passes=8, address_width=32, double_support=False, flags=0),
        # an odd size, double_support bytes of a 64-bit host, the host build's jitter order
        dict(name="passes-hy-637x359", kind="passes", geometry="hy", width=637, height=359, objects=77, hops=7,
             passes=5, address_width=64, double_support=True, flags=_lib.HTC_FLAG_JITTER_YX),
        # the scene of the hy example: four tiled objects
        dict(name="example-hy-800x600", kind="example", geometry="hy", width=800, height=600, objects=4, hops=3,
             passes=16, address_width=32),
        # many tiled objects
        dict(name="example-hy-1080p", kind="example", geometry="hy", width=1920, height=1080, objects=64, hops=8,
             passes=4, address_width=32),
        # the scene of the eu example: gradient background, refraction
        dict(name="example-eu-800x600", kind="example", geometry="eu", width=800, height=600, objects=3, hops=4,
             passes=16, address_width=32),
        # the mixed batch: every size and object count of batch.config3 together
        dict(name="batch-24-views", kind="batch", views=24, passes=6),
        # a burst of requests: seven interactive frames to three batch jobs
        dict(name="serve-12-requests", kind="serve", requests=12, passes=8),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "passes", "passes", "passes", "example", "batch", "serve"])
    if kind == "batch":
        return dict(kind=kind, views=rng.randint(6, 23), passes=rng.randint(2, 6))
    if kind == "serve":
        return dict(kind=kind, requests=rng.randint(4, 11), passes=rng.randint(2, 8))
    geometry = rng.choice(["eu", "hy", "hy"])
    width = _log(rng, 250, 1920)
    height = max(180, min(1080, int(width * rng.uniform(0.5, 0.8))))
    case = dict(kind=kind, geometry=geometry, width=width, height=height, hops=rng.randint(3, 8),
                address_width=rng.choice([32, 64]))
    if kind == "example":
        case["objects"] = _log(rng, 5, 64) if geometry == "hy" else _log(rng, 4, 16)
    else:
        case["objects"] = _log(rng, 12, 200) if geometry == "hy" else _log(rng, 5, 33)
        case["double_support"] = rng.random() < 0.25
        case["flags"] = rng.choice([0, 0, _lib.HTC_FLAG_JITTER_YX])
    if kind != "frame":   # 4e5 to 1.6e7 samples
        case["passes"] = max(2, min(64, _log(rng, 4e5, 1.6e7) // (width * height)))
    return case


# ----------------------------------------------------------------------------- inputs

def _camera_eu(rng):
    return B.random_hom3(rng)


def _scene(case, seed):
    """The view's scene: the generators of the repository's workloads, any object count."""
    rng = np.random.default_rng(seed + 7)
    n = case["objects"]
    if case["geometry"] == "eu":
        return S.euclidean_scene(n - 1, case["hops"], seed, camera=_camera_eu(rng))
    # few objects: planes mostly and near (config1); many: horospheres mostly, farther (config2)
    far = n > 40
    horo = int(round((0.6 if far else 1 / 3) * n))
    return S.hyperbolic_scene(n - horo, horo, 6.0 if far else 3.0, case["hops"], seed, camera=S.random_moebius(rng, 0.5))


def _example_value(case, seed):
    rng = np.random.default_rng(seed + 7)
    if case["geometry"] == "hy":
        if case["objects"] == 4:
            return T.hy_example_value(S.mo_chain(T.hy_example_camera(), V.geodesic_step(rng, 0.2)))
        return T.hy_tiled_random_value(seed, case["objects"], 3.0)
    if case["objects"] == 3:
        return T.eu_example_value((tuple(np.array([0.0, 0.5, 2.0]) + rng.uniform(-0.2, 0.2, 3)), (1.0, 0.0, 0.0, 0.0)))
    return T.eu_gradient_random_value(seed, case["objects"])


def _views(n, seed):
    """Views of batch.config3, the sizes and geometries in turn so that every batch has them all."""
    rng = np.random.default_rng(seed)
    pool = B.config3(seed=seed, n_views=n)
    sizes = [(256, 256), (640, 480), (1280, 720), (1920, 1080)]
    for i, v in enumerate(pool):
        v.width, v.height = sizes[(i // 2) % len(sizes)]
        v.global_seed = int(rng.integers(1 << 31))
    return pool


def _request(scene, width, height, passes, seed, interactive, image):
    data = np.frombuffer(scene.to_bytes(), dtype=np.uint8).copy()
    req = _lib.HtcRequest(data.ctypes.data, len(data), width, height, scene.recipe, scene.hops, 0, 32, passes, seed,
                          _lib.HTC_PRIORITY_INTERACTIVE if interactive else _lib.HTC_PRIORITY_BATCH, 4, GAMMA, 0,
                          image.data_ptr(), None, None)
    return req, data


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("frame", "passes"):
        ctx = P.Context(0, P.Config(case["address_width"], case["double_support"]))
        scene = _scene(case, seed)
        size = (case["width"], case["height"])
        if kind == "frame":
            return dict(kind=kind, pipeline=P.Pipeline(ctx, size, scene, flags=case["flags"], global_seed=seed))
        return dict(kind=kind, render=P.Render(ctx, scene.recipe, scene.hops, case["flags"]),
                    scene=P.EntityBuffer(ctx, scene), canvas=P.Canvas(ctx, size, seed), passes=case["passes"])
    if kind == "example":
        ctx = P.Context(0, P.Config(case["address_width"]))
        hy = case["geometry"] == "hy"
        return dict(kind=kind, passes=case["passes"], canvas=P.Canvas(ctx, (case["width"], case["height"]), seed),
                    render=P.Render(ctx, _lib.HTC_RECIPE_HY_TILED if hy else _lib.HTC_RECIPE_EU_GRADIENT, case["hops"]),
                    scene=P.EntityBuffer(ctx, _example_value(case, seed), T.hy_tiled_type() if hy else T.eu_gradient_type()))
    ctx = P.Context(0)
    if kind == "batch":
        views = _views(case["views"], seed)
        for v in views:
            v.allocate(ctx)
        renderer = B.BatchRenderer(ctx)
        passes = [1 + (i * 5) % case["passes"] for i in range(len(views))]
        renderer.set_views(views, passes)
        return dict(kind=kind, renderer=renderer, views=views, passes=passes)
    server = V.Server(ctx, hbm_budget_bytes=16 << 30)
    requests, images = [], []
    for i, v in enumerate(_views(case["requests"], seed)):
        interactive = i % 10 < 7
        w, h = (1280, 720) if interactive else (v.width, v.height)
        images.append(torch.empty((h, w, 4), dtype=torch.uint8, pin_memory=True))
        requests.append(_request(v.scene, w, h, case["passes"], v.global_seed, interactive, images[-1]))
    return dict(kind=kind, server=server, requests=requests, images=images)


# ----------------------------------------------------------------------------- one pass

def _serve(state):
    server, stream = state["server"], state["server"].ctx.stream()
    rid, rendered, n = ctypes.c_uint64(), ctypes.c_uint32(), ctypes.c_uint32()
    ids = (ctypes.c_uint64 * 256)()
    for req, _ in state["requests"]:
        _lib.call("htc_server_submit", server.handle, ctypes.byref(req), ctypes.byref(rid))
    done = 0
    while done < len(state["requests"]):
        _lib.call("htc_server_step", server.handle, stream, ctypes.byref(rendered))
        _lib.call("htc_server_poll", server.handle, ids, len(ids), ctypes.byref(n), 0 if rendered.value else 1)
        done += n.value
    return state["images"]


def run(state):
    kind = state["kind"]
    if kind == "frame":
        p = state["pipeline"]
        p.render()
        return dict(image=p.get_image(), canvas=p.canvas.image, seeds=p.canvas.seeds)
    if kind in ("passes", "example"):
        canvas = state["canvas"]
        state["render"].render_passes(state["scene"], canvas, state["passes"], sync=False)
        return dict(canvas=canvas.image, seeds=canvas.seeds)
    if kind == "batch":
        state["renderer"].render()
        return [dict(canvas=v.canvas.image, seeds=v.canvas.seeds) for v in state["views"]]
    return _serve(state)


# ----------------------------------------------------------------------------- what it cannot do without

# Floating-point operations of one executed hop without any search for the object that is hit:
# the maps into its frame and back for the test and again for the material (the ray maps of
# transform/moebius.cc: 256 each, of chain.inl: 70), the shape test and the material.
HOP_FLOPS = {"hy": 4 * 256 + 90, "eu": 4 * 70 + 70}


def _hops(h):
    """Hops of a path when a fifth of the surfaces end it (the workloads' share of emitters)."""
    return (1 - 0.8 ** h) / 0.2


def _view_work(geometry, width, height, objects, hops, passes, image):
    px = width * height
    # scene in, canvas and seeds in and out, and the packed image out where it is asked for
    return (128 * objects + px * (2 * 16 + 2 * 4 + (4 if image else 0)), px * passes * _hops(hops) * HOP_FLOPS[geometry])


def work(case):
    if case["kind"] in ("batch", "serve"):
        n = case["views"] if case["kind"] == "batch" else case["requests"]
        parts = []
        for i in range(n):   # mean object count of the pool's hyperbolic views: 110
            geometry = "eu" if i % 2 == 0 else "hy"
            w, h = [(256, 256), (640, 480), (1280, 720), (1920, 1080)][(i // 2) % 4]
            passes = 1 + (i * 5) % case["passes"]
            if case["kind"] == "serve":
                w, h = (1280, 720) if i % 10 < 7 else (w, h)
                passes = case["passes"]
            parts.append(_view_work(geometry, w, h, 9 if geometry == "eu" else 110, 4 if geometry == "eu" else 8,
                                    passes, case["kind"] == "serve"))
    else:
        parts = [_view_work(case["geometry"], case["width"], case["height"], case["objects"], case["hops"],
                            case.get("passes", 1), case["kind"] == "frame")]
    return dict(bytes=sum(p[0] for p in parts), flops=sum(p[1] for p in parts))


# ----------------------------------------------------------------------------- in 64 bits
# The Euclidean views in FP64: the samples follow the same random numbers, so a pixel differs only
# by rounding, and by a branch where rounding decides one. Hyperbolic paths have no such value:
# 3-10 % of them take another branch in 64 bits than in 32 (rays diverge exponentially), far more
# than rounding alone moves any of the others.

EPS = 1e-6


def _fmix(h):
    h = h ^ (h >> 16)
    h = (h * 0x85EBCA6B) & 0xFFFFFFFF
    h = h ^ (h >> 13)
    h = (h * 0xC2B2AE35) & 0xFFFFFFFF
    return h ^ (h >> 16)


class _Rng:
    def __init__(self, state):
        self.state = state

    def draw(self, who):
        self.state = torch.where(who, (self.state * 1103515245 + 12345) & 0xFFFFFFFF, self.state)
        return self.state.double() / 4294967296.0


def _dot(a, b):
    return (a * b).sum(-1)


def _unit(a):
    return a / a.norm(dim=-1, keepdim=True)


def _rotate(q, p):
    """q (0, p) q* for one quaternion (real part first) and many points."""
    w, u = q[0], q[1:].expand_as(p)
    t = torch.linalg.cross(u, p) * 2
    return p * (w * w + (q[1:] ** 2).sum()) + w * t + torch.linalg.cross(u, t)


def _hemisphere(u0, u1, n):
    """The cosine sample (phi from u0, cos^2 from u1) about n, turned as rot3_look_at(-n) turns +z."""
    s, c = (1 - u1).sqrt(), u1.sqrt()
    r = torch.stack([torch.cos(2 * math.pi * u0) * s, torch.sin(2 * math.pi * u0) * s, c], -1)
    d = -n
    flip = d[:, 2] >= 0
    d = torch.where(flip[:, None], -d, d)
    r = torch.where(flip[:, None], torch.stack([r[:, 0], -r[:, 1], -r[:, 2]], -1), r)   # half a turn about x first
    c = ((1 - d[:, 2]) / 2).sqrt()
    u = torch.stack([d[:, 1], -d[:, 0], torch.zeros_like(c)], -1) / (2 * c)[:, None]   # cross(-z, d) / 2c
    t = torch.linalg.cross(u, r) * 2
    return r + c[:, None] * t + torch.linalg.cross(u, t)


def _quadratic(p, v, again):
    b = -_dot(v, p)
    d = 1 - ((p + v * b[:, None]) ** 2).sum(-1)
    root = d.clamp(min=0).sqrt()
    w = torch.where(again, EPS, -EPS)
    near = torch.where(b - root < w, b + root, b - root)
    return torch.where((d < 0) | (near < w), -1.0, near)


def _plane(p, v, again):
    return torch.where(again | (p[:, 2] * v[:, 2] > 0), -1.0, -p[:, 2] / v[:, 2])


def _slabs(p, v):
    a, b = (-1 - p) / v, (1 - p) / v
    return torch.minimum(a, b), torch.maximum(a, b)


def _cube(p, v, again):
    lo, hi = _slabs(p, v)
    near, far = lo.amax(-1), hi.amin(-1)
    w = torch.where(again, 2 * EPS, -2 * EPS)
    t = torch.where(near < w, far, near)
    return torch.where((near > far) | (t < w), -1.0, t)


def _cube_normal(p, v, t):
    """Outward normal of the face that p + t v lies on."""
    h = p + v * t[:, None]
    axis = h.abs().argmax(-1, keepdim=True)
    return torch.zeros_like(h).scatter_(-1, axis, torch.sign(h.gather(-1, axis)))


SHAPES = {"plane": _plane, "sphere": _quadratic, "cube": _cube}


def _f32(x):
    return torch.tensor(np.asarray(x, dtype=np.float64).astype(np.float32).astype(np.float64), device="cuda")


def _objects(case, seed):
    """(camera shift, camera rotation, fov, background, objects) with every number rounded as it is serialized."""
    one = [1.0, 0.0, 0.0, 0.0]
    if case["kind"] == "example":
        value = _example_value(case, seed)
        shift, rot = value["view"]["map"]
        bg = value["background"]
        objects = []
        for o in value["object"]:
            m, shape = o["inner"]["material"], o["inner"]["shape"][0].lower()
            parts = [("diffuse", m["diffuse"]["portion"], m["diffuse"]["material"]["color"], 0.0),
                     ("specular", m["specular"]["portion"], None, 0.0),
                     ("refractive", m["refractive"]["portion"], m["refractive"]["material"]["color"],
                      m["refractive"]["material"]["inner"]["index"])]
            objects.append((_f32(o["map"]), _f32(one), shape, parts))
        return (_f32(shift), _f32(rot), value["view"]["inner"]["fov"],
                (_f32(bg["direction"]), _f32(bg["colors"][0]), _f32(bg["colors"][1]), float(np.float32(bg["power"]))), objects)
    scene = _scene(case, seed)
    objects = []
    for o in scene.objects:
        m = o.material
        parts = [("diffuse", m.diffuse, m.diffuse_color, 0.0), ("specular", m.specular, None, 0.0),
                 ("emission", m.luminous, m.emission, 0.0)]
        objects.append((_f32(o.map.shift), _f32(o.map.rot), "plane" if o.shape == S.SHAPE_PLANE else "sphere", parts))
    return _f32(scene.camera.shift), _f32(scene.camera.rot), scene.fov, (_f32(scene.background),), objects


def _interact(parts, rng, who, n, v, light, out, go):
    """The mixture of one object for the paths `who` (normal n, local direction v)."""
    alpha = rng.draw(who)
    left = who
    for kind, portion, color, index in parts:
        alpha = alpha - float(np.float32(portion))
        mine = left & (alpha < 0)
        left = left & ~mine
        if kind == "emission":
            out += torch.where(mine[:, None], light * _f32(color), 0.0)
            continue
        if color is not None:
            light *= torch.where(mine[:, None], _f32(color), 1.0)
        if kind == "diffuse":
            u0, u1 = rng.draw(mine), rng.draw(mine)
            to = _hemisphere(u0, u1, torch.where((_dot(v, n) > 0)[:, None], -n, n))
        elif kind == "specular":
            to = v - 2 * _dot(v, n)[:, None] * n
        else:
            a = _dot(v, n)
            k = torch.where(a < -EPS, 1 / float(np.float32(index)), float(np.float32(index)))
            x = (a * a - 1) * k * k + 1
            bend = torch.sign(a) * x.clamp(min=0).sqrt() - a * k
            to = torch.where((x > EPS)[:, None], v * k[:, None] + bend[:, None] * n, v - 2 * a[:, None] * n)
        v = torch.where(mine[:, None], to, v)
        go |= mine
    return v


def _sample(case, cam, objects, rng, px, py, size):
    shift, rot, fov, bg = cam
    every = torch.ones_like(px, dtype=torch.bool)
    u0, u1 = rng.draw(every), rng.draw(every)
    jx, jy = (u1, u0) if case.get("flags", 0) & _lib.HTC_FLAG_JITTER_YX else (u0, u1)
    v = _unit(torch.stack([px + size * (jx - 0.5), py + size * (jy - 0.5), torch.full_like(px, -1 / fov)], -1))
    v, p = _rotate(rot, v), shift.expand_as(v).clone()
    out, light = torch.zeros_like(p), torch.ones_like(p)
    alive, last = every, torch.full(px.shape, -1, dtype=torch.long, device=px.device)
    for _ in range(case["hops"]):
        best, which = torch.full_like(px, -1.0), torch.full_like(last, -1)
        for k, (s, q, shape, _parts) in enumerate(objects):
            back = torch.cat([q[:1], -q[1:]])
            t = SHAPES[shape](_rotate(back, p - s), _unit(_rotate(back, v)), last == k)
            nearer = (t > -EPS) & ((best <= -EPS) | (t < best))
            best, which = torch.where(nearer, t, best), torch.where(nearer, k, which)
        miss = alive & (which < 0)
        if len(bg) == 1:
            sky = bg[0].expand_as(out)
        else:
            f = (0.5 * (_dot(v, bg[0].expand_as(v)) + 1)).clamp(0, 1)[:, None] ** bg[3]
            sky = f * bg[1] + (1 - f) * bg[2]
        out += torch.where(miss[:, None], sky * light, 0.0)
        go = torch.zeros_like(alive)
        for k, (s, q, shape, parts) in enumerate(objects):
            who = alive & (which == k)
            back = torch.cat([q[:1], -q[1:]])
            lp, lv = _rotate(back, p - s), _unit(_rotate(back, v))
            if shape == "plane":
                n = torch.zeros_like(lp)
                n[:, 2] = -1
            elif shape == "sphere":
                n = _unit(lp + lv * best[:, None])
            else:
                n = _cube_normal(lp, lv, best)
            hit = lp + lv * best[:, None]
            to = _interact(parts, rng, who, n, lv, light, out, go)
            p = torch.where(who[:, None], _rotate(q, hit) + s, p)
            v = torch.where(who[:, None], _unit(_rotate(q, to)), v)
        last = torch.where(go, which, last)
        alive = go
    return out


def exact(case, seed):
    if case["kind"] not in ("frame", "passes", "example") or case["geometry"] != "eu":
        return None
    w, h, passes = case["width"], case["height"], case.get("passes", 1)
    if w * h * passes * case["objects"] * case["hops"] > 6e9:   # about 20 seconds
        return None
    shift, rot, fov, bg, objects = _objects(case, seed)
    i = torch.arange(w * h, device="cuda")
    rng = _Rng(_fmix((seed & 0xFFFFFFFF) ^ _fmix(i)))
    px, py = (2 * (i % w) + 1 - w).double() / h, (h - 2 * (i // w) - 1).double() / h
    canvas = torch.zeros((w * h, 4), dtype=torch.float64, device="cuda")
    for _ in range(passes):
        canvas[:, :3] += _sample(case, (shift, rot, float(np.float32(fov)), bg), objects, rng, px, py, 2.0 / h)
        canvas[:, 3] += 1
    canvas = canvas.reshape(-1)
    return dict(image=None, canvas=canvas, seeds=None) if case["kind"] == "frame" else dict(canvas=canvas, seeds=None)
