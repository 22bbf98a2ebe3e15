"""The calls a program makes of this framework, as measurable cases.

Two seeded scenes carry them: "small" (64 primitives in a 32 m cube at 4 cm)
and "large" (512 primitives in a 256 m cube at 2 cm, ~1.1 million bricks),
both with every primitive drawn from the case's seed.  A renderer marches
views into device planes on its own stream; a physics step asks distances at
points; a shading pass takes shadow and ambient-occlusion rays from the
views' hits; an editor edits and looks at the result; a server answers a mix
of requests from host buffers.

``exact`` restates the march and the queries over the small scene in 64-bit
torch, from the primitives alone.  The large scene has no such value: its
four thousand million brick centres and thousand-step rays would take minutes
in plain torch.
"""
from __future__ import annotations

import ctypes as C
import dataclasses
import math
import random

import numpy as np
import torch

from rkifield_b200 import _abi as abi
from rkifield_b200 import engine, scenes

SPECS = {"small": scenes.SCENE_SMALL, "large": scenes.SCENE_LARGE}
POOL = {"small": 80_000, "large": 2_000_000}  # brick slots a program reserves
MODES = {"closest": abi.RKF_TRACE_CLOSEST, "any": abi.RKF_TRACE_ANY, "shadow": abi.RKF_TRACE_SHADOW}
STRATEGIES = {"brute": abi.RKF_STRATEGY_BRUTE, "tiled": abi.RKF_STRATEGY_TILED, "bvh": abi.RKF_STRATEGY_BVH}
MAX_FLOAT = 3.402823e38


def listed():
    return [
        # a physics step: one frame's contact points, from host memory
        {"name": "points_host_300", "kind": "points", "scene": "small", "n": 300, "mem": "host"},
        # the largest point query the server takes, on the device
        {"name": "points_65536", "kind": "points", "scene": "large", "n": 65536, "mem": "device"},
        # ambient occlusion at the visible points of a 960x540 shading pass
        {"name": "ao_points_200003", "kind": "ao", "scene": "small", "n": 200_003},
        # the smallest image in use: a thumbnail of the small scene, f32 distances
        {"name": "view_256x256_f32", "kind": "view", "scene": "small", "precision": "f32", "w": 256, "h": 256,
         "strategy": "brute", "extra": 0, "planes": False},
        # the engine's default internal resolution, with the reference G-buffer planes
        {"name": "view_960x540_large", "kind": "view", "scene": "large", "precision": "f16", "w": 960, "h": 540,
         "strategy": "brute", "extra": 0, "planes": True},
        # the headline view
        {"name": "view_1920x1080_large", "kind": "view", "scene": "large", "precision": "f16", "w": 1920, "h": 1080,
         "strategy": "brute", "extra": 0, "planes": False},
        # the least memory: u8 distances, the whole small scene in view
        {"name": "view_1920x1080_u8", "kind": "view", "scene": "small", "precision": "u8", "w": 1920, "h": 1080,
         "strategy": "brute", "extra": 0, "planes": False},
        # several objects under the tiled strategy, as the runtime binds it, at an odd window size
        {"name": "view_1277x717_tiled", "kind": "view", "scene": "small", "precision": "f16", "w": 1277, "h": 717,
         "strategy": "tiled", "extra": 4, "planes": True},
        # a ray-cast batch: random origins and directions
        {"name": "rays_250007_large", "kind": "rays", "scene": "large", "precision": "f16", "n": 250_007,
         "mode": "closest"},
        # a frame of four views with their shadow and ambient-occlusion rays
        {"name": "frame_4_views", "kind": "frame", "scene": "large", "views": "173x97,343x193,661x372,1280x720",
         "lights": 4, "ao": 8},
        # an editor's largest stroke and the view that shows it
        {"name": "edit_and_view", "kind": "edit", "scene": "large", "radius": 1.0, "w": 960, "h": 540},
        # a burst of mixed requests to the serving loop
        {"name": "serve_48", "kind": "serve", "scene": "large", "requests": 48},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, lo, hi):
    """Width and height of an image of lo to hi pixels, 16:9 or a square."""
    px = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    w = max(8, int(round(math.sqrt(px * (16.0 / 9.0 if rng.random() < 0.75 else 1.0)))))
    return w, max(8, int(round(px / w)))


def draw(rng: random.Random):
    kind = rng.choice(["points", "ao", "view", "view", "view", "rays", "rays", "frame", "edit", "serve"])
    scene = rng.choice(["small", "large"])
    if kind == "points":
        return {"kind": kind, "scene": scene, "n": _log_int(rng, 32, 65536), "mem": rng.choice(["host", "device"])}
    if kind == "ao":
        return {"kind": kind, "scene": scene, "n": _log_int(rng, 64, 500_000)}
    if kind == "view":
        multi = rng.random() < 0.35
        w, h = _size(rng, 64 ** 2, 1277 * 717 if multi else 1920 * 1080)
        return {"kind": kind, "scene": scene, "precision": rng.choice(["f16", "f16", "f32", "u8"]), "w": w, "h": h,
                "strategy": rng.choice(["brute", "tiled", "bvh"]) if multi else "brute",
                "extra": rng.randint(1, 6) if multi else 0, "planes": rng.random() < 0.5}
    if kind == "rays":
        return {"kind": kind, "scene": scene, "precision": rng.choice(["f16", "f16", "f32", "u8"]),
                "n": _log_int(rng, 64, 1 << 20), "mode": rng.choice(["closest", "any", "shadow"])}
    if kind == "frame":
        views = ",".join("%dx%d" % _size(rng, 128 ** 2, 300_000) for _ in range(rng.randint(1, 4)))
        return {"kind": kind, "scene": scene, "views": views, "lights": rng.randint(1, 4), "ao": rng.choice([2, 4, 8])}
    w, h = _size(rng, 64 ** 2, 960 * 540)
    if kind == "edit":
        return {"kind": kind, "scene": scene, "radius": round(rng.uniform(0.1, 1.0), 3), "w": w, "h": h}
    return {"kind": kind, "scene": scene, "requests": rng.randint(8, 48)}


# --------------------------------------------------------------------------
# Inputs
# --------------------------------------------------------------------------
_stream = None


def _frame_stream():
    """The one stream a program records its frames on."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    return _stream.cuda_stream


def _spec(case, seed):
    return dataclasses.replace(SPECS[case["scene"]], seed=1000 + seed)


def _rng(seed, salt):
    return np.random.default_rng([seed, salt])


def _dev(n, dtype):
    return torch.zeros(n, dtype=dtype, device="cuda")


def _planes(n, reference=False):
    g = {"t": _dev(n, torch.float32), "normal": _dev(3 * n, torch.float32), "slot": _dev(n, torch.int32),
         "material": _dev(n, torch.int16), "flags": _dev(n, torch.int16)}
    if reference:
        g.update(position=_dev(4 * n, torch.float32), packed_material=_dev(n, torch.int32),
                 motion=_dev(4 * n, torch.float32))
    return g


def _ptrs(d):
    return {k: v.data_ptr() for k, v in d.items()}


def _gb(d):
    g = abi.rkf_gbuffer()
    for k, v in d.items():
        setattr(g, k, v.data_ptr())
    g.mem = abi.RKF_MEM_DEVICE
    return g


def _hits(d):
    h = abi.rkf_hits()
    for k, v in d.items():
        setattr(h, k, v.data_ptr())
    h.mem = abi.RKF_MEM_DEVICE
    return h


def _context(spec, case, seed):
    prims = scenes.make_prims(spec)
    ctx = engine.Context(pool_capacity=POOL[case["scene"]], precision=case.get("precision", "f16"),
                         keep_reference_pool=False, max_inflight=256, mem_budget_bytes=2 << 30)
    ctx.voxelize(prims, scenes.voxelize_params(spec, prims))
    return ctx, prims


def _with_analytic(ctx, spec, rng, n):
    """The voxelized object beside n analytic ones (spheres, boxes, capsules)
    in front of the scene, as a world with props."""
    objs = [ctx.object(0)]
    for i in range(n):
        o = abi.rkf_gpu_object()
        c = rng.uniform(-0.4, 0.4, 3) * spec.cube
        for a in range(4):
            o.inverse_world[5 * a] = 1.0
        kind = i % 3
        size = rng.uniform(0.5, 2.0, 3)
        par = [size[0], 0.0, 0.0, 0.0] if kind == 0 else [*size, 0.0] if kind == 1 else [size[0], size[1], 0.0, 0.0]
        o.sdf_params[:] = [float(x) for x in par]
        r = float(np.sum(size))
        for a in range(3):
            o.inverse_world[12 + a] = -float(c[a])
            o.aabb_min[a], o.aabb_max[a] = float(c[a]) - r, float(c[a]) + r
            o.accumulated_scale[a] = 1.0
        o.sdf_type, o.primitive_type = abi.RKF_SDF_ANALYTICAL, (abi.RKF_PRIM_SPHERE, abi.RKF_PRIM_BOX,
                                                                abi.RKF_PRIM_CAPSULE)[kind]
        o.material_id, o.object_id = 40 + i, 2 + i
        objs.append(o)
    ctx.update_objects(objs, [0] + [-1] * n)
    return objs


def _camera(spec, case, seed, w, h):
    if case["scene"] == "large":
        return scenes.seeded_camera(spec, w, h, seed=100 + seed, inside=True, distance=spec.cube * 0.18)
    return scenes.seeded_camera(spec, w, h, seed=11 + seed)


def _near_view(prims, rng, w, h):
    """A camera a few metres from a primitive, looking at it."""
    p = prims[int(rng.integers(0, len(prims)))]
    c = p["centre"].astype(np.float64)
    u = rng.standard_normal(3)
    u /= np.linalg.norm(u)
    return scenes.camera_uniforms(c + (float(p["bound_radius"]) + rng.uniform(2.0, 8.0)) * u, c, w, h)


def _query_points(case, seed, spec, prims):
    """Half of the points anywhere in the scene, half near its surfaces."""
    half = 0.5 * spec.cube
    pts = _rng(seed, 1).uniform(-half, half, (case["n"], 3)).astype(np.float32)
    pts[::2] = _surface_points(case, seed, prims)[0][::2]
    return pts


def _surface_points(case, seed, prims):
    """Points just off the primitives' surfaces, with outward directions."""
    rng = _rng(seed, 2)
    p = prims[rng.integers(0, len(prims), case["n"])]
    u = rng.standard_normal((case["n"], 3))
    u /= np.linalg.norm(u, axis=1, keepdims=True)
    c = p["centre"].astype(np.float64)
    pos = c + u * (p["params"][:, :1].astype(np.float64) + 0.08)
    return pos.astype(np.float32), u.astype(np.float32)


def _rays(case, seed, spec):
    rng = _rng(seed, 3)
    half, n = 0.5 * spec.cube, case["n"]
    o = rng.uniform(-half, half, (n, 3)).astype(np.float32)
    d = rng.standard_normal((n, 3))
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
    return o, d, np.full(n, 32.0, np.float32)


def _cuda(a):
    return torch.from_numpy(np.ascontiguousarray(a)).reshape(-1).cuda()


class _Serving:
    """A serving session and the page-locked buffers of a burst of requests."""

    def __init__(self, ctx, spec, prims, p, rng, n):
        self.ctx = ctx
        half = 0.5 * spec.cube
        self.reqs = []
        sizes = random.Random(n)  # the mix of kinds and sizes is the case's, what is in them the seed's
        for _ in range(n):
            kind = sizes.randrange(3)
            if kind == 0:
                px = math.exp(sizes.uniform(math.log(64 ** 2), math.log(640 * 360)))
                w = max(16, int(round(math.sqrt(px * 16.0 / 9.0))))
                h = max(9, int(round(w * 9.0 / 16.0)))
                self.reqs.append((0, w * h, (_near_view(prims, rng, w, h), w, h)))
            elif kind == 1:
                m = _log_int(sizes, 1, 1 << 17)
                o = rng.uniform(-half, half, (m, 3)).astype(np.float32)
                d = rng.standard_normal((m, 3))
                d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
                self.reqs.append((1, m, (o, d, np.full(m, 32.0, np.float32))))
            else:
                m = _log_int(sizes, 1, 65536)
                self.reqs.append((2, m, (rng.uniform(-half, half, (m, 3)).astype(np.float32),)))
        rays = sum(m for k, m, _ in self.reqs if k < 2)
        pts = sum(m for k, m, _ in self.reqs if k == 2)
        pin = lambda m, dt: torch.zeros(max(1, m), dtype=dt, pin_memory=True)  # noqa: E731
        self.out = {"t": pin(rays, torch.float32), "normal": pin(3 * rays, torch.float32),
                    "slot": pin(rays, torch.int32), "material": pin(rays, torch.int16),
                    "flags": pin(rays, torch.int16), "dist": pin(pts, torch.float32),
                    "grad": pin(3 * pts, torch.float32), "point_material": pin(pts, torch.int16)}
        self.keep = []
        self.work = []
        view = {k: v.numpy() for k, v in self.out.items()}
        at_r = at_p = 0
        for kind, m, args in self.reqs:
            if kind == 2:
                o = {"dist": view["dist"][at_p:at_p + m], "grad": view["grad"][3 * at_p:3 * (at_p + m)],
                     "material": view["point_material"][at_p:at_p + m]}
                at_p += m
            else:
                o = {"t": view["t"][at_r:at_r + m], "normal": view["normal"][3 * at_r:3 * (at_r + m)],
                     "slot": view["slot"][at_r:at_r + m], "material": view["material"][at_r:at_r + m],
                     "flags": view["flags"][at_r:at_r + m]}
                at_r += m
            if kind:
                pinned = [torch.from_numpy(np.ascontiguousarray(a).reshape(-1)).pin_memory() for a in args]
                self.keep.append(pinned)
                args = [x.numpy() for x in pinned]
            self.work.append((kind, args, o))
        self.server = engine.Server(ctx, p)

    def burst(self):
        tickets = []
        for kind, a, o in self.work:
            if kind == 0:
                tickets.append(self.server.submit_render(*a, o))
            elif kind == 1:
                tickets.append(self.server.submit_rays(*a, abi.RKF_TRACE_CLOSEST, o))
            else:
                tickets.append(self.server.submit_points(*a, o))
        for t in tickets:
            while self.server.poll(t, 1_000_000) is None:
                pass
        return self.out

    def __del__(self):
        try:
            self.server.stop()
            self.ctx.close()
        except Exception:
            pass


def prepare(case, seed):
    spec = _spec(case, seed)
    kind = case["kind"]
    ctx, prims = _context(spec, case, seed)
    p = scenes.march_params(spec)
    s = {"kind": kind, "ctx": ctx, "p": p}
    if kind == "points":
        pts = _query_points(case, seed, spec, prims)
        s["host"] = case["mem"] == "host"
        if s["host"]:
            s["pts"] = pts
        else:
            n = case["n"]
            s.update(pts=_cuda(pts), n=n, dist=_dev(n, torch.float32), grad=_dev(3 * n, torch.float32),
                     material=_dev(n, torch.int16))
    elif kind == "ao":
        pos, nrm = _surface_points(case, seed, prims)
        s.update(pos=_cuda(pos), nrm=_cuda(nrm), n=case["n"], out=_dev(case["n"], torch.float32))
    elif kind == "view":
        w, h = case["w"], case["h"]
        if case["extra"]:
            objs = _with_analytic(ctx, spec, _rng(seed, 4), case["extra"])
            if case["strategy"] == "bvh":
                ctx.upload_bvh(engine.object_bvh(objs))
        p.strategy = STRATEGIES[case["strategy"]]
        s.update(cam=_camera(spec, case, seed, w, h), w=w, h=h, out=_planes(w * h, case["planes"]))
        if case["scene"] == "large" and not case["extra"]:
            # the launch tuning the autotuner finds for such a view, kept from an earlier session
            ctx.set_tuning(abi.rkf_batch_tuning(8, 4, 64, 128, 0, 256, 32, 0, 0, 1, 0))
    elif kind == "rays":
        o, d, t = _rays(case, seed, spec)
        n = case["n"]
        out = {"t": _dev(n, torch.float32), "flags": _dev(n, torch.int16)}
        if case["mode"] == "closest":
            out.update(normal=_dev(3 * n, torch.float32), slot=_dev(n, torch.int32), material=_dev(n, torch.int16))
        s.update(o=_cuda(o), d=_cuda(d), tmax=_cuda(t), n=n, mode=MODES[case["mode"]], out=out)
    elif kind == "frame":
        _prepare_frame(s, case, seed, prims)
    elif kind == "edit":
        rng = _rng(seed, 6)
        w, h = case["w"], case["h"]
        q = prims[int(rng.integers(0, len(prims)))]
        c = q["centre"].astype(np.float64)
        u = rng.standard_normal(3)
        u /= np.linalg.norm(u)
        at = c + u * float(q["params"][0])
        ops = []
        for edit_type in (0, 1):  # a sphere added, then carved out again
            op = abi.rkf_edit_op()
            op.edit_type, op.falloff, op.strength, op.blend_k, op.material_id = edit_type, 1, 1.0, 0.05, 17
            op.position[:] = [float(x) for x in at]
            op.rotation[:] = (0.0, 0.0, 0.0, 1.0)
            op.dimensions[:] = (case["radius"], 0.0, 0.0)
            ops.append(op)
        cam = scenes.camera_uniforms(at + 5.0 * u, at, w, h)
        s.update(ops=ops, turn=0, cam=cam, w=w, h=h, out=_planes(w * h))
    else:
        s["serving"] = _Serving(ctx, spec, prims, p, _rng(seed, 7), case["requests"])
    return s


def _prepare_frame(s, case, seed, prims):
    rng = _rng(seed, 5)
    sizes = [tuple(int(x) for x in v.split("x")) for v in case["views"].split(",")]
    nv, nl, na = len(sizes), case["lights"], case["ao"]
    views, batches = (abi.rkf_view * nv)(), (abi.rkf_ray_batch * (2 * nv))()
    s.update(views=views, batches=batches, nv=nv, nl=nl, na=na, seed=seed & 0xFFFF, gb=[], rays=[], hits=[],
             sec=[], lights=[])
    for i, (w, h) in enumerate(sizes):
        n = w * h
        cam = _near_view(prims, rng, w, h)
        g = _planes(n)
        views[i].camera, views[i].width, views[i].height, views[i].out = cam, w, h, _gb(g)
        target = np.array(cam.position[:3], np.float64) + 8.0 * np.array(cam.forward[:3], np.float64)
        lights = (target[None] + rng.uniform(-10, 10, (nl, 3)) + np.array([0.0, 8.0, 0.0])).astype(np.float32)
        rays, outs = [], []
        for j, (per, mode) in enumerate(((nl, abi.RKF_TRACE_SHADOW), (na, abi.RKF_TRACE_ANY))):
            r = [_dev(3 * per * n, torch.float32), _dev(3 * per * n, torch.float32), _dev(per * n, torch.float32)]
            o = {"t": _dev(per * n, torch.float32), "flags": _dev(per * n, torch.int16)}
            b = batches[2 * i + j]
            b.origins, b.dirs, b.tmax = (x.data_ptr() for x in r)
            b.n, b.mode, b.out = per * n, mode, _hits(o)
            rays += r
            outs.append(o)
        s["gb"].append(g)
        s["rays"].append(rays)
        s["sec"].append(outs)
        s["lights"].append(lights)


# --------------------------------------------------------------------------
# One pass
# --------------------------------------------------------------------------
def run(s):
    ctx, p, kind = s["ctx"], s["p"], s["kind"]
    lib, stream = ctx.lib, _frame_stream()
    if kind == "points":
        if s["host"]:
            d, g, m = ctx.query_points(s["pts"])
            return {"dist": d, "grad": g, "material": m.view(np.int16)}
        abi.check(lib.rkf_query_points(ctx.h, s["pts"].data_ptr(), s["n"], s["dist"].data_ptr(), s["grad"].data_ptr(),
                                       s["material"].data_ptr(), abi.RKF_MEM_DEVICE), "rkf_query_points")
        return {"dist": s["dist"], "grad": s["grad"], "material": s["material"]}
    if kind == "ao":
        abi.check(lib.rkf_sdf_ao(ctx.h, s["pos"].data_ptr(), s["nrm"].data_ptr(), s["n"], s["out"].data_ptr(),
                                 abi.RKF_MEM_DEVICE), "rkf_sdf_ao")
        return s["out"]
    if kind == "view":
        ctx.march_async(s["cam"], p, s["w"], s["h"], _ptrs(s["out"]), stream)
        return s["out"]
    if kind == "rays":
        h = _hits(s["out"])
        abi.check(lib.rkf_trace_rays(ctx.h, s["o"].data_ptr(), s["d"].data_ptr(), s["tmax"].data_ptr(), s["n"],
                                     s["mode"], C.byref(p), abi.RKF_MEM_DEVICE, C.byref(h)), "rkf_trace_rays")
        return s["out"]
    if kind == "frame":
        return _run_frame(s, stream)
    if kind == "edit":
        op = s["ops"][s["turn"] & 1]
        s["turn"] += 1
        ctx.edit(op)
        ctx.march_async(s["cam"], p, s["w"], s["h"], _ptrs(s["out"]), stream)
        return s["out"]
    return s["serving"].burst()


def _run_frame(s, stream):
    ctx, p = s["ctx"], s["p"]
    lib, nv = ctx.lib, s["nv"]
    abi.check(lib.rkf_march_batch_async(ctx.h, s["views"], nv, None, 0, C.byref(p), None, stream), "views")
    hit = []
    for i in range(nv):
        v, n = s["views"][i], C.c_uint32()
        abi.check(lib.rkf_secondary_rays(ctx.h, C.byref(v.camera), v.width, v.height, C.byref(v.out),
                                         s["lights"][i].ctypes.data, s["nl"], s["na"], 1.0, s["seed"] + i,
                                         *[x.data_ptr() for x in s["rays"][i]], C.byref(n), stream), "secondary")
        hit.append(int(n.value))
    abi.check(lib.rkf_march_batch_async(ctx.h, None, 0, s["batches"], 2 * nv, C.byref(p), None, stream), "secondary")
    return {"views": s["gb"], "rays": s["rays"], "secondary": s["sec"], "hits": hit}


# --------------------------------------------------------------------------
# What a pass cannot do without
# --------------------------------------------------------------------------
def work(case):
    """Inputs read once and outputs written once.  Operations: a ray or a point
    cannot do without one distance (its grid coordinates, eight corners and
    seven mixes: 60), a point's gradient without six more, a ray of a view
    without its direction (40)."""
    kind = case["kind"]
    if kind == "points":
        return {"bytes": case["n"] * (12 + 4 + 12 + 2), "flops": case["n"] * 7 * 60}
    if kind == "ao":
        return {"bytes": case["n"] * (24 + 4), "flops": case["n"] * 4 * 70}
    if kind == "view":
        n = case["w"] * case["h"]
        return {"bytes": n * (24 + (36 if case["planes"] else 0)), "flops": n * 100}
    if kind == "rays":
        return {"bytes": case["n"] * (28 + (24 if case["mode"] == "closest" else 6)), "flops": case["n"] * 60}
    if kind == "frame":
        n = 0
        for v in case["views"].split(","):
            w, h = (int(x) for x in v.split("x"))
            n += w * h
        sec = n * (case["lights"] + case["ao"])
        # each secondary ray is written once and read once (28 bytes) and answered (6)
        return {"bytes": n * (24 + 18) + sec * (28 + 28 + 6), "flops": (n + sec) * 100}
    if kind == "edit":
        n = case["w"] * case["h"]
        vox = (2 * case["radius"] / SPECS[case["scene"]].voxel_size) ** 3
        return {"bytes": n * 24 + vox * 10, "flops": n * 100 + vox * 100}
    return {"bytes": case["requests"] * 24 * 20_000, "flops": case["requests"] * 100 * 20_000}


# --------------------------------------------------------------------------
# The same in 64 bits, from the primitives
# --------------------------------------------------------------------------
class _Grid:
    """The small scene's voxelized object in 64-bit torch: bricks of the
    narrow band with their voxel values at the stored precision."""

    def __init__(self, spec, precision):
        f32 = lambda x: float(np.float32(x))  # noqa: E731
        self.prims = scenes.make_prims(spec)
        vp = scenes.voxelize_params(spec, self.prims)
        self.vs = f32(vp.voxel_size)
        self.be = f32(np.float32(self.vs) * np.float32(8))
        self.k, self.cut = f32(vp.smooth_k), f32(vp.cut_distance)
        band = f32(np.float32(vp.band_voxels) * np.float32(self.vs))
        self.dims = [max(1, int(math.ceil(float((np.float32(vp.aabb_max[a]) - np.float32(vp.aabb_min[a]))
                                                / np.float32(self.be))))) for a in range(3)]
        self.gs = torch.tensor([d * self.be for d in self.dims], dtype=torch.float64, device="cuda")
        dx, dy, dz = self.dims
        flat = torch.arange(dx * dy * dz, device="cuda")
        b = torch.stack([flat % dx, (flat // dx) % dy, flat // (dx * dy)], 1)
        lo = b.double() * self.be - self.gs / 2
        centre = self.sdf(lo + self.be / 2)
        thr = band + self.be * 0.8660254 + self.vs
        index = torch.where(centre > 0, -1, -2)  # EMPTY, INTERIOR, else a brick
        cand = torch.nonzero(centre.abs() <= thr)[:, 0]
        v = torch.arange(512, device="cuda")
        off = (torch.stack([v & 7, (v >> 3) & 7, v >> 6], 1).double() + 0.5) * self.vs
        values, count = [], 0
        for part in cand.split(8192):
            d = self.sdf((lo[part][:, None] + off[None]).reshape(-1, 3)).reshape(-1, 512)
            keep = (d.abs() <= band).any(1) | ~((d > 0).all(1) | (d < 0).all(1))
            index[part] = torch.where((d > 0).all(1), -1, -2)
            index[part[keep]] = torch.arange(count, count + int(keep.sum()), device="cuda")
            count += int(keep.sum())
            values.append(self.stored(d[keep], band, precision))
        self.index, self.values = index, torch.cat(values).reshape(-1)
        own = b[index >= 0].double()
        self.gmin = own.min(0).values * self.be - self.gs / 2
        self.gmax = (own.max(0).values + 1) * self.be - self.gs / 2

    def sdf(self, q):
        acc = torch.full((q.shape[0],), math.inf, dtype=torch.float64, device="cuda")
        for p in self.prims:
            c = torch.tensor(p["centre"].astype(np.float64), device="cuda")
            r = q - c
            near = (r.norm(dim=1) - float(p["bound_radius"])) < self.cut
            if not bool(near.any()):
                continue
            loc = r[near] @ torch.tensor(p["rot"].reshape(3, 3).astype(np.float64), device="cuda")
            a = [float(x) for x in p["params"]]
            if p["type"] == scenes.PRIM_SPHERE:
                d = loc.norm(dim=1) - a[0]
            elif p["type"] == scenes.PRIM_BOX:
                e = loc.abs() - torch.tensor(a, dtype=torch.float64, device="cuda")
                d = e.clamp_min(0).norm(dim=1) + e.max(1).values.clamp_max(0)
            else:
                loc = loc.clone()
                loc[:, 1] -= loc[:, 1].clamp(-a[1], a[1])
                d = loc.norm(dim=1) - a[0]
            old = acc[near]
            h = (self.k - (old - d).abs()).clamp_min(0) / self.k
            acc[near] = torch.minimum(old, d) - h * h * self.k * 0.25
        return acc

    def stored(self, d, band, precision):
        if precision == "f16":
            return d.half().double()
        if precision == "f32":
            return d.float().double()
        a = d.abs()
        step = a.max(1, keepdim=True).values.clamp(1e-6, 3.0 * self.vs) / 127.0
        return torch.sign(d) * (a / step).floor().clamp_max(127) * step

    def sample(self, l, grad=False):
        """The trilinear sampler at object-local positions (n, 3)."""
        gp = l + self.gs / 2
        lo = 0.01 * self.vs
        cl = torch.minimum(gp.clamp_min(lo), self.gs - lo)
        outside = (gp - cl).norm(dim=1)
        vc = cl / self.vs - 0.5
        f = vc.floor()
        t = vc - f
        i0 = f.long()
        top = torch.tensor(self.dims, device="cuda") * 8 - 1
        c = [torch.minimum(i0.clamp_min(0), top), torch.minimum((i0 + 1).clamp_min(0), top)]
        d = torch.zeros_like(outside)
        for k in range(8):
            s = [(k >> a) & 1 for a in range(3)]
            x = torch.stack([c[s[a]][:, a] for a in range(3)], 1)
            w = 1.0
            for a in range(3):
                w = w * (t[:, a] if s[a] else 1 - t[:, a])
            b = x >> 3
            e = self.index[b[:, 0] + b[:, 1] * self.dims[0] + b[:, 2] * self.dims[0] * self.dims[1]]
            at = e.clamp_min(0) * 512 + (x[:, 0] & 7) + (x[:, 1] & 7) * 8 + (x[:, 2] & 7) * 64
            v = torch.where(e >= 0, self.values[at],
                            torch.where(e == -1, self.be, -self.be if grad else -2 * self.vs))
            d = d + w * v
        d = d + outside
        if not grad:
            g = (l - torch.minimum(torch.maximum(l, self.gmin), self.gmax)).norm(dim=1)
            d = torch.where(g > self.be, g, d)
        return torch.where(outside > 2 * self.be, outside, d)

    def gradient(self, q):
        e = 2 * self.vs
        g = torch.stack([self.sample(q + e * u, True) - self.sample(q - e * u, True)
                         for u in torch.eye(3, dtype=torch.float64, device="cuda")], 1)
        n = g.norm(dim=1, keepdim=True)
        up = torch.tensor([0.0, 1.0, 0.0], dtype=torch.float64, device="cuda")
        return torch.where(n < 1e-10, up, g / n)

    def march(self, o, d, tmax, p, mode):
        """t (or the shadow factor) and normal of each ray."""
        n = o.shape[0]
        z = lambda x: torch.full((n,), x, dtype=torch.float64, device="cuda")  # noqa: E731
        shadow = mode == "shadow"
        t, prev_t, prev_d, out = z(0.005 if shadow else 0.0), z(0.0), z(MAX_FLOAT), z(1.0 if shadow else MAX_FLOAT)
        near, crossed = z(0.0), torch.zeros(n, dtype=torch.bool, device="cuda")
        live = t <= tmax
        hit = torch.zeros_like(live)
        hi_t = z(0.0)
        near_max = 32 if shadow else p.scene.max_steps
        for _ in range(256 if shadow else p.hard_max_steps):
            i = torch.nonzero(live)[:, 0]
            if not len(i):
                break
            b = self.sample(o[i] + d[i] * t[i, None])
            if shadow:
                blocked = b < 0.005
                out[i[blocked]] = 0.0
                pen = ~blocked & (b < 0.02)
                out[i[pen]] = torch.minimum(out[i[pen]], 16.0 * b[pen] / t[i[pen]])
                near[i[pen]] += 1
                stop, step = blocked, b.clamp_min(0.005)
            else:
                over = (b < 0) & (prev_d[i] > p.scene.hit_threshold)
                stop = over | (b < p.scene.hit_threshold)
                hit[i[stop]] = True
                crossed[i[over]] = True
                near[i[~stop & (b < p.near_surface_threshold)]] += 1
                step = b.clamp_min(p.min_step)
            go = i[~stop]
            prev_t[go], prev_d[go] = t[go], b[~stop]
            t[go] += step[~stop]
            live[i[stop]] = False
            live &= (t <= tmax) & (near < near_max)
        if shadow:
            return out.clamp(0, 1), None
        if mode == "closest":
            i = torch.nonzero(crossed)[:, 0]
            lo, hi = prev_t[i], t[i]
            for _ in range(p.bisect_steps):
                mid = (lo + hi) / 2
                inside = self.sample(o[i] + d[i] * mid[:, None]) < 0
                lo, hi = torch.where(inside, lo, mid), torch.where(inside, mid, hi)
            t[i] = (lo + hi) / 2
        i = torch.nonzero(hit)[:, 0]
        out[i] = t[i]
        normal = torch.zeros((n, 3), dtype=torch.float64, device="cuda")
        if mode == "closest" and len(i):
            normal[i] = self.gradient(o[i] + d[i] * t[i, None])
        return out, normal


def exact(case, seed):
    kind = case["kind"]
    if case["scene"] != "small" or kind not in ("points", "ao", "view", "rays"):
        return None  # the large scene: minutes in plain torch; frames, edits and servers march many such views
    if kind == "view" and case["extra"]:
        return None  # which skips a ray takes depends on binary16 texels, not on numbers that 64 bits refine
    spec = _spec(case, seed)
    g = _Grid(spec, case.get("precision", "f16"))
    p = scenes.march_params(spec)
    f64 = lambda a: torch.from_numpy(np.asarray(a)).double().cuda()  # noqa: E731
    if kind == "points":
        q = f64(_query_points(case, seed, spec, g.prims))
        return {"dist": g.sample(q), "grad": g.gradient(q).reshape(-1), "material": None}
    if kind == "ao":
        pos, nrm = (f64(a) for a in _surface_points(case, seed, g.prims))
        acc = sum(0.5 ** (k - 1) * (0.12 * k - g.sample(pos + nrm * (0.12 * k))) for k in range(1, 5))
        return (1.0 - 0.7 * acc).clamp(0, 1)
    if kind == "rays":
        o, d, tmax = (f64(a) for a in _rays(case, seed, spec))
        t, normal = g.march(o, d, tmax, p, case["mode"])
        out = {"t": t, "flags": None}
        if case["mode"] == "closest":
            out.update(normal=normal.reshape(-1), slot=None, material=None)
        return out
    w, h = case["w"], case["h"]
    cam = _camera(spec, case, seed, w, h)
    i = torch.arange(w * h, device="cuda")
    u, v = ((i % w).double() + 0.5) / w, ((i // w).double() + 0.5) / h
    axes = [f64(np.array(list(a)[:3], np.float64)) for a in (cam.forward, cam.right, cam.up, cam.position)]
    d = axes[0] + (2 * u - 1)[:, None] * axes[1] + (1 - 2 * v)[:, None] * axes[2]
    d = d / d.norm(dim=1, keepdim=True)
    o = axes[3].expand(w * h, 3)
    tmax = torch.full((w * h,), float(p.scene.max_distance), dtype=torch.float64, device="cuda")
    t, normal = g.march(o, d, tmax, p, "closest")
    out = {"t": t, "normal": normal.reshape(-1), "slot": None, "material": None, "flags": None}
    if case["planes"]:
        hit = t < MAX_FLOAT
        pos = torch.where(hit[:, None], o + d * torch.where(hit, t, 0.0)[:, None], 0.0)
        out.update(position=torch.cat([pos, t[:, None]], 1).reshape(-1), packed_material=None, motion=None)
    return out
