"""The work that programs give this renderer, as cases to be timed and compared.

A case is one call path at one size: a frame drawn with ``draw`` (into device
memory or page-locked host memory), with ``draw_async`` or through the
``Presenter``; a batch of views replayed as one CUDA graph; or a training step
of the differentiable path (forward and backward).  ``listed()`` holds the
sizes of the repository's own configurations and tests beside smaller, larger
and ragged ones, ``draw()`` spreads over the same ranges.

Frames are compared as bytes: RGBA8, the bit patterns of the fp32 Z buffer and
the triangle count, since the renderer's contract is bit-exactness.  The
differentiable step returns its loss, image and gradients, and ``exact()``
restates it in plain torch: visibility with the reference's float32 arithmetic,
shading and adjoint in 64 bits through autograd.
"""
import dataclasses
import functools
import json
import math
import weakref

import numpy as np
import torch

import gorender_gb300 as gr
from gorender_gb300 import _native, renderer, scenes

FOV = 60.0


def listed():
    return [
        # the smallest frame a viewer draws: a 960-triangle sphere, Gouraud lit; latency and launches
        {"name": "sphere_640x360", "call": "draw", "mesh": "sphere", "n": 32, "objects": 1, "width": 640, "height": 360,
         "texture": "none", "flat": False, "marks": False, "post": False},
        # an ordinary object in a small odd window with wireframe and vertex marks, fog and crosshair
        {"name": "marks_801x599", "call": "draw", "mesh": "icosphere", "n": 5, "objects": 1, "width": 801, "height": 599,
         "texture": "none", "flat": True, "marks": True, "post": True},
        # ragged: a 20k-triangle terrain, odd window, a texture whose sides are no powers of two
        {"name": "terrain_853x479", "call": "draw", "mesh": "heightfield", "n": 101, "objects": 1, "width": 853, "height": 479,
         "texture": "odd", "flat": False, "marks": False, "post": False},
        # the headline frame, end to end into page-locked host memory (what a program without a GPU consumer does)
        {"name": "terrain_720p_host", "call": "draw_host", "mesh": "heightfield", "n": 317, "objects": 1, "width": 1280, "height": 720,
         "texture": "pow2", "flat": True, "marks": False, "post": False},
        # the same frame queued into device memory, one after the other (a frame loop feeding a GPU consumer)
        {"name": "terrain_720p_async", "call": "draw_async", "mesh": "heightfield", "n": 317, "objects": 1, "width": 1280, "height": 720,
         "texture": "pow2", "flat": True, "marks": False, "post": False},
        # the viewer's loop: an 82k-triangle textured object presented at full HD
        {"name": "present_1080p", "call": "present", "mesh": "icosphere", "n": 6, "objects": 1, "width": 1920, "height": 1080,
         "texture": "pow2", "flat": False, "marks": False, "post": False},
        # few triangles, many pixels: a textured box that fills a 4K window
        {"name": "box_2160p", "call": "draw", "mesh": "box", "n": 1, "objects": 1, "width": 3840, "height": 2160,
         "texture": "pow2", "flat": True, "marks": False, "post": False},
        # the small-triangle stress scene: 64 coloured icospheres, 5.0 M triangles
        {"name": "icospheres_1080p", "call": "draw", "mesh": "icospheres", "n": 6, "objects": 64, "width": 1920, "height": 1080,
         "texture": "none", "flat": False, "marks": False, "post": False},
        # a handful of views (thumbnails of small objects) in one replay
        {"name": "batch_8_views", "call": "batch", "views": 8, "max_tris": 5000},
        # the 256-view batch of uneven meshes at mixed resolutions
        {"name": "batch_256_views", "call": "batch", "views": 256, "max_tris": 200000},
        # a small training step: 3 views of a 1,280-face mesh, with the image, ragged sizes
        {"name": "step_3_views", "call": "step", "views": 3, "level": 3, "width": 131, "height": 97, "tex": 31, "image": True},
        # the 64-view training step of the 82k-face mesh
        {"name": "step_64_views", "call": "step", "views": 64, "level": 6, "width": 512, "height": 512, "tex": 256, "image": False},
    ]


def _spread(rng, lo, hi):
    """A whole number in [lo, hi], spread over its logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    call = rng.choice(["draw", "draw", "draw_host", "draw_async", "present", "batch", "step"])
    if call == "batch":
        return {"call": call, "views": _spread(rng, 1, 224), "max_tris": _spread(rng, 400, 200000)}
    if call == "step":
        height = _spread(rng, 48, 480)
        return {"call": call, "views": _spread(rng, 1, 56), "level": rng.randint(2, 6), "width": int(height * rng.uniform(1.0, 1.06)) + 1,
                "height": height, "tex": rng.choice([0, _spread(rng, 4, 256), _spread(rng, 4, 256)]), "image": rng.random() < 0.5}
    mesh = rng.choice(["sphere", "heightfield", "heightfield", "icosphere", "icospheres", "box"])
    n = {"sphere": _spread(rng, 5, 200), "heightfield": _spread(rng, 4, 900), "icosphere": rng.randint(1, 7),
         "icospheres": rng.randint(3, 6), "box": 1}[mesh]
    width = _spread(rng, 100, 3600)
    height = max(40, int(width * rng.uniform(0.4, 0.6)))
    return {"call": call, "mesh": mesh, "n": n, "objects": _spread(rng, 2, 60) if mesh == "icospheres" else 1, "width": width, "height": height,
            "texture": rng.choice(["none", "pow2", "odd"]), "flat": rng.random() < 0.5, "marks": mesh in ("sphere", "icosphere", "box") and rng.random() < 0.25, "post": rng.random() < 0.15}


# ---- scenes ----

_icosphere = functools.lru_cache(maxsize=None)(scenes.icosphere)


def _box():
    """A unit cube: 8 vertices, 12 faces, corner UVs."""
    p = np.array([[x, y, z, 1.0] for x in (-1, 1) for y in (-1, 1) for z in (-1, 1)], np.float32)
    quads = [(1, 5, 7, 3), (4, 0, 2, 6), (0, 1, 3, 2), (5, 4, 6, 7), (2, 3, 7, 6), (0, 4, 5, 1)]
    f, uv = [], []
    for a, b, c, d in quads:
        f += [(a, b, c), (a, c, d)]
        uv += [(0, 0, 1, 0, 1, 1), (0, 0, 1, 1, 0, 1)]
    return scenes.MeshData(pos=p, vidx=np.array(f, np.int32), uv=np.array(uv, np.float32), name="box")


def _frame_scene(case, seed):
    """Objects, camera and texture of a frame; the seed turns, bends and colours them."""
    rng = np.random.default_rng(seed)
    turn = tuple(float(x) for x in rng.uniform(-0.4, 0.4, 3))
    flags = scenes.DEFAULT_FLAGS | (scenes.FLAT_SHADING if case["flat"] else 0)
    if case["marks"]:
        flags |= scenes.SHOW_EDGES | scenes.SHOW_VERTICES
    if case["post"]:
        flags |= renderer.CROSSHAIR
    camera = scenes.CameraData((0.0, 0.0, 3.0), (0.0, 0.0, -1.0), (0.0, 1.0, 0.0))
    objects, kind, n = [], case["mesh"], case["n"]
    if kind == "sphere":
        m = scenes.uv_sphere(n, max(3, n // 2))
    elif kind == "heightfield":
        # the camera stands inside the terrain's extent: faces cross the near and the side planes
        m = scenes.heightfield(n, seed=seed)
        turn = (0.0, turn[1] * 0.2, 0.0)
        camera = scenes.CameraData((0.3, 0.35, 2.5), (0.0, -0.3, -1.0), (0.0, 1.0, 0.0))
        if not case["flat"]:
            vn = np.zeros((m.nv, 4), np.float32)
            vn[:, 1] = vn[:, 3] = 1.0
            vn[:, [0, 2]] = rng.uniform(-0.2, 0.2, (m.nv, 2))
            m.vnrm, m.nidx = vn, m.vidx.copy()
    elif kind == "box":
        m = _box()
        turn = tuple(0.2 * t for t in turn)
        camera = scenes.CameraData((0.1, 0.05, 1.9), (0.0, 0.0, -1.0), (0.0, 1.0, 0.0))
    else:
        m = _icosphere(n)
        if kind == "icosphere":
            pos = m.pos.copy()
            pos[:, :3] *= (1.0 + rng.uniform(-0.05, 0.05, (m.nv, 1))).astype(np.float32)
            m = dataclasses.replace(m, pos=pos)
    textures = []
    if case["texture"] != "none":
        w, h = (16, 16) if case["texture"] == "pow2" else (23, 17)
        textures = [scenes.random_texture(w, h, seed=seed + 1, scale=8.0)]
        m = dataclasses.replace(m, tex=np.zeros(m.nf, np.int32), uv=m.uv if m.uv is not None else scenes.spherical_uvs(m))
    if kind == "icospheres":
        # spheres of a level and the one below it in a 40-unit cube, with their own vertex colours
        small = _icosphere(max(1, n - 1))
        camera = scenes.CameraData((0.0, 0.0, 0.0), (0.0, 0.0, -1.0), (0.0, 1.0, 0.0))
        few = set(rng.permutation(case["objects"])[: max(1, case["objects"] // 16)].tolist())
        for k in range(case["objects"]):
            base = small if k in few else m
            if base is small and textures:
                base = dataclasses.replace(small, tex=np.zeros(small.nf, np.int32), uv=scenes.spherical_uvs(small))
            mesh = dataclasses.replace(base, vcolor=rng.random((base.nv, 3), dtype=np.float32))
            p, s = rng.uniform(-20.0, 20.0, 3), float(rng.uniform(0.2, 2.0))
            objects.append(scenes.ObjectData(mesh, (s, s, s), (0.0, 0.0, 0.0), (float(p[0]), float(p[1]), float(p[2]) - 30.0)))
    else:
        objects = [scenes.ObjectData(m, (1.0, 1.0, 1.0), turn, (0.0, 0.0, 0.0))]
    return scenes.SceneData(kind, case["width"], case["height"], objects, camera, textures, flags, FOV)


# A program has one context per device: the scenes of one case share it, and
# their asynchronous frames follow each other on its one stream.
_contexts = weakref.WeakValueDictionary()


def _context(case):
    key = json.dumps(case, sort_keys=True)
    ctx = _contexts.get(key)
    if ctx is None:
        ctx = gr.Context(0)
        _contexts[key] = ctx
        if case.get("post"):
            ctx.set_fog(True, 0.9, 0.2, (90, 100, 120, 255))
    return ctx


class _Scene(gr.UploadedScene):
    """An uploaded scene that gives its meshes back when the program drops it."""

    def __del__(self):
        if self.ctx.handle:
            for h in set(self.mesh_handles):
                _native.lib().gr_mesh_destroy(self.ctx.handle, h)


class _Frame(np.ndarray):
    """A presented frame in the presenter's page-locked memory, which it keeps alive."""

    presenter = None


def _frame_state(case, seed):
    scene = _frame_scene(case, seed)
    ctx = _context(case)
    s = {"call": case["call"], "up": _Scene(ctx, scene), "n": len(scene.objects)}
    w, h = case["width"], case["height"]
    if case["call"] == "present":
        r = gr.Renderer(ctx, w, h)
        r.set_fov(gr.fov_radians(scene.fov_deg))
        _native.check(_native.lib().gr_renderer_set_flags(r._h, scene.flags))
        s["objects"] = [gr.Object(k, o.scale, o.rotation, o.translation) for k, o in zip(s["up"].mesh_handles, scene.objects)]
        s["camera"] = gr.Camera(scene.camera.position, scene.camera.direction, scene.camera.up)
        s["presenter"] = gr.Presenter(r)
        s["presenter"].frame(s["objects"], s["camera"], copy=False)  # the loop is running: each call returns the frame before
    else:
        where = {"pin_memory": True} if case["call"] == "draw_host" else {"device": "cuda"}
        s["rgba"] = torch.zeros((h, w, 4), dtype=torch.uint8, **where)
        s["z"] = torch.zeros((h, w), dtype=torch.float32, **where)
        torch.cuda.synchronize()
        # the first frame sizes the context's buffers: an asynchronous one cannot be drawn again by itself
        gr.draw(ctx, s["up"].items, s["n"], s["up"].params, s["rgba"].data_ptr(), s["z"].data_ptr())
    return s


def _batch_state(case, seed):
    ctx = gr.Context(0)
    ups, views, entries, at = [], [], [], 0
    specs = scenes.multiview_batch(case["views"], seed=seed, max_tris=case["max_tris"])
    # the seed makes meshes and poses; the resolutions go round, so that every batch of a case has the same outputs
    sizes = ((256, 256), (512, 512), (640, 360), (1280, 720))
    specs = [dataclasses.replace(sc, width=sizes[k // 2 % 4][0], height=sizes[k // 2 % 4][1]) for k, sc in enumerate(specs)]
    for sc in specs:
        at += (sc.width * sc.height + 63) // 64 * 64
    rgba = torch.zeros((at, 4), dtype=torch.uint8, device="cuda")
    z = torch.zeros((at,), dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    at = 0
    for v, sc in enumerate(specs):
        up = gr.UploadedScene(ctx, sc)
        views.append((up.params, rgba.data_ptr() + 4 * at, z.data_ptr() + 4 * at))
        entries += [(h, m[0], m[1], v) for h, m in zip(up.mesh_handles, up.matrices)]
        at += (sc.width * sc.height + 63) // 64 * 64
    return {"call": "batch", "ctx": ctx, "batch": renderer.Batch(ctx, views, entries, autotune=True), "rgba": rgba, "z": z}


def _step_inputs(case, seed):
    """Mesh, parameters, views and target of a training step."""
    sc = scenes.diff_scene(views=case["views"], size=8, level=case["level"], tex_size=max(1, case["tex"]), seed=seed)
    sc = dataclasses.replace(sc, width=case["width"], height=case["height"])
    world, views = renderer.diff_views(sc)
    g = torch.Generator("cuda").manual_seed(seed)
    target = torch.rand((case["views"], case["height"], case["width"], 4), generator=g, device="cuda") * 0.6
    params = {"pos": sc.mesh.pos, "vcol": sc.vcol, "tex": sc.tex, "light": sc.light}
    return sc.mesh, world, views, params, target


def _step_state(case, seed):
    mesh, world, views, params, target = _step_inputs(case, seed)
    ctx = gr.Context(0)
    if not case["tex"]:
        mesh = dataclasses.replace(mesh, uv=None)
    s = {"call": "step", "ctx": ctx, "target": target, "light": params["light"]}
    s["diff"] = renderer.Diff(ctx, ctx.mesh(mesh), world, views, tex_size=(case["tex"], case["tex"]))
    for k in ("pos", "vcol", "tex"):
        s[k] = torch.from_numpy(params[k]).cuda() if k != "tex" or case["tex"] else None
        s["g_" + k] = None if s[k] is None else torch.zeros_like(s[k])
    s["image"] = torch.zeros_like(target) if case["image"] else None
    torch.cuda.synchronize()
    return s


def prepare(case, seed):
    if case["call"] == "batch":
        return _batch_state(case, seed)
    if case["call"] == "step":
        return _step_state(case, seed)
    return _frame_state(case, seed)


def _ptr(t):
    return None if t is None else t.data_ptr()


def run(s):
    if s["call"] == "present":
        rgba, tpf = s["presenter"].frame(s["objects"], s["camera"], copy=False)
        rgba = rgba.view(_Frame)
        rgba.presenter = s["presenter"]
        return {"rgba": rgba, "tpf": tpf}
    if s["call"] == "batch":
        s["batch"].run()
        s["batch"].sync()  # a replay whose buffers overflowed is run again here
        return {"rgba": s["rgba"], "z": s["z"].view(torch.int32)}
    if s["call"] == "step":
        tex = s["tex"]
        loss = s["diff"].forward(s["pos"].data_ptr(), s["vcol"].data_ptr(), _ptr(tex), s["light"], s["target"].data_ptr(), _ptr(s["image"]))
        light = s["diff"].backward(s["g_pos"].data_ptr(), s["g_vcol"].data_ptr(), _ptr(s["g_tex"]))
        out = {"loss": loss, "light": torch.from_numpy(light).float(), "pos": s["g_pos"], "vcol": s["g_vcol"]}
        if tex is not None:
            out["tex"] = s["g_tex"]
        if s["image"] is not None:
            out["image"] = s["image"]
        return out
    up = s["up"]
    if s["call"] == "draw_async":
        gr.draw_async(up.ctx, up.items, s["n"], up.params, s["rgba"].data_ptr(), s["z"].data_ptr())
        return {"rgba": s["rgba"], "z": s["z"].view(torch.int32)}
    tpf = gr.draw(up.ctx, up.items, s["n"], up.params, s["rgba"].data_ptr(), s["z"].data_ptr())
    return {"rgba": s["rgba"], "z": s["z"].view(torch.int32), "tpf": tpf}


# ---- what a pass cannot do without ----

def _mesh_size(kind, n):
    """(vertices, faces) of a mesh."""
    if kind == "sphere":
        lat = max(3, n // 2)
        return n * (lat - 1) + 2, 2 * n * (lat - 1)
    if kind == "heightfield":
        return n * n, 2 * (n - 1) ** 2
    if kind == "box":
        return 8, 12
    return 10 * 4 ** n + 2, 20 * 4 ** n


def work(case):
    if case["call"] == "batch":
        # the means of the ranges that the views are drawn from (log-uniform faces, four resolutions)
        faces = case["views"] * (case["max_tris"] - 100) / math.log(case["max_tris"] / 100)
        pixels = case["views"] * (256 * 256 + 512 * 512 + 640 * 360 + 1280 * 720) / 4
        verts = faces / 2
        return {"bytes": 16 * verts + (12 + 16 + 8) * faces + 8 * pixels, "flops": 60 * verts + 60 * faces + 30 * pixels}
    if case["call"] == "step":
        v, f = _mesh_size("icosphere", case["level"])
        px = case["views"] * case["width"] * case["height"]
        # parameters, indices and normals once a step; target in, image out; gradients out
        mesh = v * (16 + 12) + f * 24 + v * 16 + (f * 24 + 16 * case["tex"] ** 2 if case["tex"] else 0)
        grads = v * (16 + 12) + 16 * case["tex"] ** 2
        return {"bytes": mesh + grads + px * (16 + (16 if case["image"] else 0)), "flops": case["views"] * (60 * v + 60 * f) + 400 * px}
    v, f = _mesh_size(case["mesh"] if case["mesh"] != "icospheres" else "icosphere", case["n"])
    v, f = v * case["objects"], f * case["objects"]
    px = case["width"] * case["height"]
    lit = 16 * f if case["flat"] or case["mesh"] == "box" else 16 * v + 12 * f
    tex = 24 * f if case["texture"] != "none" else 12 * v if case["mesh"] == "icospheres" else 0
    out = 4 if case["call"] == "present" else 8
    return {"bytes": 16 * v + 12 * f + lit + tex + out * px, "flops": 60 * v + 60 * f + 30 * px}


# ---- the training step in plain torch ----

def _visible(pos, vidx, mvp, screen, width, height):
    """The face that the reference's raster leaves at each pixel (-1: none) of one view whose faces all lie inside the frustum, in its float32 arithmetic."""
    def row(m, r, x, y, z, w):
        return ((m[4 * r] * x + m[4 * r + 1] * y) + m[4 * r + 2] * z) + m[4 * r + 3] * w

    m, sc = [float(x) for x in mvp], [float(x) for x in screen]
    c = [row(m, r, pos[:, 0], pos[:, 1], pos[:, 2], pos[:, 3]) for r in range(4)]
    d = [x / c[3] for x in c]
    sx, sy = (row(sc, r, *d).long() for r in (0, 1))
    f = [vidx[:, k] for k in range(3)]
    # facingCamera on the clip-space corners
    p = [[c[r][f[k]] for r in range(3)] for k in range(3)]
    e1, e2 = ([p[k][r] - p[0][r] for r in range(3)] for k in (1, 2))
    nx, ny, nz = e1[1] * e2[2] - e1[2] * e2[1], e1[2] * e2[0] - e1[0] * e2[2], e1[0] * e2[1] - e1[1] * e2[0]
    facing = (nx * (0.0 - p[0][0]) + ny * (0.0 - p[0][1])) + nz * (0.0 - p[0][2]) > 0
    x, y, w = [sx[k] for k in f], [sy[k] for k in f], [c[3][k] for k in f]
    a, b, e = [], [], []
    for i, j in ((0, 1), (1, 2), (2, 0)):
        dx, dy = y[i] - y[j], x[j] - x[i]
        keep = (dy > 0) | ((dy == 0) & (dx > 0))
        a.append(dx), b.append(dy), e.append(x[i] * y[j] - x[j] * y[i] - (~keep).long())
    total = e[0] + e[1] + e[2]
    x0, x1 = torch.stack(x).amin(0).clamp(min=0), torch.stack(x).amax(0).clamp(max=width - 1)
    y0, y1 = torch.stack(y).amin(0).clamp(min=0), torch.stack(y).amax(0).clamp(max=height - 1)
    live = torch.nonzero(facing & (total < 0) & (x0 <= x1) & (y0 <= y1))[:, 0]
    bw, bh = (x1 - x0 + 1)[live], (y1 - y0 + 1)[live]
    own = torch.repeat_interleave(torch.arange(len(live), device=pos.device), bw * bh)
    at = torch.arange(len(own), device=pos.device) - (torch.cumsum(bw * bh, 0) - bw * bh)[own]
    t = live[own]
    px, py = x0[t] + at % bw[own], y0[t] + at // bw[own]
    ev = [a[k][t] * px + b[k][t] * py + e[k][t] for k in range(3)]
    inside = torch.nonzero((ev[0] < 0) & (ev[1] < 0) & (ev[2] < 0))[:, 0]
    t, px, py, e12, e20 = t[inside], px[inside], py[inside], ev[1][inside].float(), ev[2][inside].float()
    s = total[t].float()
    al, be = e12 / s, e20 / s
    ga = (1.0 - al) - be
    z = -((al / w[0][t] + be / w[1][t]) + ga / w[2][t])
    ok = z > 0  # every corner lies in front of the camera
    key = (z.view(torch.int32).long() << 32) | (t + 1)
    best = torch.zeros(width * height, dtype=torch.int64, device=pos.device)
    best.scatter_reduce_(0, (py * width + px)[ok], key[ok], "amax")
    return (best & 0xFFFFFFFF) - 1


def exact(case, seed):
    if case["call"] != "step":
        return None  # frames are bytes, bit patterns and counts
    mesh, world, views, params, target = _step_inputs(case, seed)
    dev, f64 = target.device, torch.float64
    pos32, vidx = torch.from_numpy(mesh.pos).to(dev), torch.from_numpy(mesh.vidx).long().to(dev)
    nidx, uv = torch.from_numpy(mesh.nidx).long().to(dev), torch.from_numpy(mesh.uv).to(dev)
    pos, vcol, tex, light = (torch.from_numpy(params[k]).to(dev, f64).requires_grad_() for k in ("pos", "vcol", "tex", "light"))
    n = torch.from_numpy(mesh.vnrm).to(dev, f64) @ torch.from_numpy(np.asarray(world, np.float64).reshape(4, 4).T).to(dev)
    nhat = n[:, :3] / n.norm(dim=1, keepdim=True)
    loss, images, size = 0.0, [], case["tex"]
    for k, (width, height, _, screen, mvp) in enumerate(views):
        ids = _visible(pos32, vidx, mvp, screen, width, height)
        hit = torch.nonzero(ids >= 0)[:, 0]
        S, M = (torch.from_numpy(np.asarray(m, np.float64).reshape(4, 4)).to(dev) for m in (screen, mvp))
        q = torch.stack([(S @ M)[0], (S @ M)[1], M[3]])
        h = torch.cat([pos[:, :3], pos[:, 3:].detach()], 1) @ q.T  # homogeneous screen x, y and clip W
        v = vidx[ids[hit]]
        px, py = (hit % width).to(f64), torch.div(hit, width, rounding_mode="floor").to(f64)
        c = h[v]
        a, b, w = c[..., 0] - px[:, None] * c[..., 2], c[..., 1] - py[:, None] * c[..., 2], c[..., 2]
        D = torch.stack([a[:, (i + 1) % 3] * b[:, (i + 2) % 3] - a[:, (i + 2) % 3] * b[:, (i + 1) % 3] for i in range(3)], 1)
        T = D.sum(1)
        m = (D * torch.where(T < 0, -1.0, 1.0)[:, None]).clamp(min=0)
        ok = (w < 0).all(1) & (T != 0) & (m.sum(1) > 0)
        hit, v, m = hit[ok], v[ok], m[ok]
        face = ids[hit]
        l = m / m.sum(1, keepdim=True)
        I = (l * (0.5 + 0.5 * (nhat[nidx[face]] * light).sum(-1))).sum(1)
        col = (l[..., None] * vcol[v]).sum(1)
        if size:
            # the texel is chosen from float32 barycentrics and coordinates
            m32 = m.detach().float()
            l0, l1 = (m32[:, j] / ((m32[:, 0] + m32[:, 1]) + m32[:, 2]) for j in range(2))
            t = uv[face].view(-1, 3, 2)
            st = (l0[:, None] * t[:, 0] + l1[:, None] * t[:, 1]) + ((1.0 - l0) - l1)[:, None] * t[:, 2]
            st = torch.floor(st * float(size)).long() % size
            t = tex[st[:, 1], st[:, 0]]
        else:
            t = torch.ones((len(hit), 4), dtype=f64, device=dev)
        out = torch.zeros((width * height, 4), dtype=f64, device=dev)
        out = out.index_put((hit,), torch.cat([(I[:, None] * col) * t[:, :3], t[:, 3:]], 1))
        part = (out - target[k].view(-1, 4).to(f64)).square().sum()
        part.backward()
        loss += float(part.detach())
        images.append(out.detach().view(height, width, 4))
    g = {"loss": torch.tensor(loss, dtype=f64), "light": light.grad, "pos": torch.cat([pos.grad[:, :3], torch.zeros_like(pos.grad[:, 3:])], 1),
         "vcol": vcol.grad}
    if size:
        g["tex"] = tex.grad
    if case["image"]:
        g["image"] = torch.stack(images)
    return g
