"""The differentiable kernels where they branch, against the FP64 adjoint of
the oracle: normals indexed apart from the vertices, meshes without UVs, sizes that
leave a CTA's blocks of pixels partly outside (small views take 8 rows a CTA,
2^21 pixels and more 64), views of different sizes, a position gradient
buffer that is not 16-byte aligned, and losses beyond float32."""
import dataclasses

import numpy as np
import pytest

import gorender_gb300 as gr
from gorender_gb300 import renderer as R
from oracle import oracle
from tests import diff_cases as dc

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

GRAD_TOL, LOSS_TOL = 1e-4, 1e-5  # the bounds of the differentiable path's own tests


def _records(diff):
    _, rec, n = diff.buffers()

    class Dev:
        __cuda_array_interface__ = {"shape": (n, 4), "typestr": "<u4", "data": (rec, False), "version": 3}
    return torch.as_tensor(Dev(), device="cuda").cpu().numpy().copy()


def _ids(diff):
    ids, _, n = diff.buffers()

    class Dev:
        __cuda_array_interface__ = {"shape": (n,), "typestr": "<u4", "data": (ids, False), "version": 3}
    return torch.as_tensor(Dev(), device="cuda").cpu().numpy().copy()


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a, np.float32)).cuda()


def _step(mesh, views, world, params, target, offset=0):
    """One step: (loss, {gradients}, records).  The gradient buffers start
    `offset` floats into their allocations."""
    ctx = gr.Context(0)
    try:
        tex = params["tex"]
        d = R.Diff(ctx, ctx.mesh(mesh), world, views, tex_size=(0, 0) if tex is None else tex.shape[:2])
        p = {k: None if params[k] is None else _dev(params[k]) for k in ("pos", "vcol", "tex")}
        t = _dev(target)
        loss = d.forward(p["pos"].data_ptr(), p["vcol"].data_ptr(), None if tex is None else p["tex"].data_ptr(),
                         params["light"], t.data_ptr())
        g = {k: None if v is None else torch.zeros(v.numel() + offset * (k != "tex"), device="cuda")[offset * (k != "tex"):]
             for k, v in p.items()}
        light = d.backward(g["pos"].data_ptr(), g["vcol"].data_ptr(), None if tex is None else g["tex"].data_ptr())
        out = {k: v.cpu().numpy() for k, v in g.items() if v is not None}
        out["light"] = light
        return loss, out, _records(d)
    finally:
        ctx.close()


def _case(sizes, level, tex, seed):
    sc = dc.small_case(views=len(sizes), size=8, level=level, tex_size=max(tex, 1), seed=seed)
    fov = R.fov_radians(sc.fov_deg)
    views, world = [], None
    for (w, h), cam in zip(sizes, sc.cameras):
        mvp, world = R.object_matrices((1.0, 1.0, 1.0), (0.0, 0.0, 0.0), (0.0, 0.0, 0.0), cam.position, cam.direction,
                                       cam.up, w, h, fov)
        views.append((w, h, sc.flags, R.screen_matrix(w, h), mvp))
    params = {"pos": sc.mesh.pos, "vcol": sc.vcol, "tex": sc.tex if tex else None, "light": sc.light}
    mesh = sc.mesh if tex else dataclasses.replace(sc.mesh, uv=None)
    target = np.random.default_rng(seed).random((sum(w * h for w, h in sizes), 4), np.float32)
    return mesh, views, world, params, target


def _compare(mesh, views, world, params, target, offset=0):
    loss, g, rec = _step(mesh, views, world, params, target, offset)
    ids, texel = rec[:, 0], rec[:, 1]
    ref = oracle.diff_eval(mesh, [(w, h, s, m) for w, h, _, s, m in views], dict(params, world=world), ids, target,
                           texel_in=texel if params["tex"] is not None else None)
    assert (ids != dc.NO_FACE).sum() > 50
    assert abs(loss - ref["loss"]) <= LOSS_TOL * abs(ref["loss"])
    for k in g:
        a, b = g[k].reshape(-1), np.asarray(ref["g_" + k]).reshape(-1)
        if k == "pos":
            a, b = a.reshape(-1, 4)[:, :3], b.reshape(-1, 4)[:, :3]
            assert (g[k].reshape(-1, 4)[:, 3] == 0).all()
        assert dc.rel_err(a, b) <= GRAD_TOL, k


@pytest.mark.parametrize("sizes", [[(33, 31)], [(131, 97)] * 3, [(64, 40), (31, 65), (200, 9)]])
@pytest.mark.parametrize("tex", [0, 31])
def test_sizes(sizes, tex):
    _compare(*_case(sizes, 3, tex, seed=2))


def test_large_ragged_views():
    sizes = [(701, 603)] * 4 + [(517, 801)]
    assert sum(w * h for w, h in sizes) >= 1 << 21
    _compare(*_case(sizes, 4, 17, seed=3))


def test_normals_apart():
    mesh, views, world, params, target = _case([(131, 97)] * 2, 3, 31, seed=4)
    order = np.random.default_rng(1).permutation(mesh.nv).astype(np.int32)
    back = np.argsort(order).astype(np.int32)
    mesh = dataclasses.replace(mesh, vnrm=mesh.vnrm[order], nidx=back[mesh.vidx])
    _compare(mesh, views, world, params, target)


def test_unaligned_position_gradients():
    _compare(*_case([(131, 97)] * 2, 3, 31, seed=5), offset=1)


@pytest.mark.parametrize("value,count", [(4e18, 2000), (1e19, 3), (np.inf, 1), (np.nan, 1)])
def test_losses_beyond_float32(value, count):
    """Pixels whose squared difference nears or passes float32's largest value
    (3.4e38): the sum over many of them is a double as before; infinities and
    NaN stay."""
    mesh, views, world, params, target = _case([(131, 97)], 3, 0, seed=6)
    target[:count, 0] = value
    loss, _, _ = _step(mesh, views, world, params, target)
    one = np.float32(value) * np.float32(value)
    if np.isfinite(one):
        assert abs(loss - count * float(one)) <= 1e-6 * count * float(one)
    elif np.isnan(value):
        assert np.isnan(loss)
    else:
        assert loss == np.inf


@pytest.mark.parametrize("vertices", [1023, 1024, 1025, 2049])
@pytest.mark.parametrize("last", [(0.0, 0.0, 0.0), (-0.0, 0.0, -0.0), (0.0, 9.0, 0.0), (np.nan, 0.0, 0.0), (np.inf, 0.0, 0.0)])
def test_bounding_box_of_the_parameters(vertices, last):
    """The box takes every vertex, faces or not, in CTAs of 1024, and decides
    for each of 35 views (a warp takes a second one) what is clipped: views that
    hold the mesh, cut it, look away from it, and a box with a NaN."""
    sc = dc.small_case(views=35, size=40, level=3, tex_size=4, seed=8)
    pos = np.tile(np.array(last + (1.0,), np.float32), (vertices, 1))
    pos[:sc.mesh.nv] = sc.mesh.pos
    sc.mesh = dataclasses.replace(sc.mesh, pos=pos)
    for v, cam in enumerate(sc.cameras):
        if v % 3 == 1:
            cam.position = tuple(0.45 * x for x in cam.position)
        elif v % 3 == 2:
            cam.direction = tuple(-x for x in cam.direction)
    views, world = dc.oracle_views(sc)
    views = [(w, h, sc.flags, s, m) for w, h, s, m in views]
    ctx = gr.Context(0)
    try:
        d = R.Diff(ctx, ctx.mesh(sc.mesh), world, views, tex_size=(0, 0))
        p, vcol = _dev(pos), _dev(np.ones((vertices, 3)))
        t = _dev(np.zeros((sum(w * h for w, h, *_ in views), 4)))
        d.forward(p.data_ptr(), vcol.data_ptr(), None, sc.light, t.data_ptr())
        ids, ref = _ids(d), dc.oracle_ids(sc)
        assert (ref != dc.NO_FACE).any()
        assert np.array_equal(ids, ref)
    finally:
        ctx.close()
