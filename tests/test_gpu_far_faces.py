"""Faces with corners beyond the narrow bound (2^14 pixels), bit for bit against
the oracle: in frames with a view that does not clip k_setup takes them, in each
form of shading, with marks and without faces, at both of its register counts
(a million faces have the other) and in a batch beside a view that clips; a mesh whose
box holds a NaN passes for one inside the frustum and is not clipped at all."""
import dataclasses

import numpy as np
import pytest

import gorender_gb300 as gr
from gorender_gb300 import renderer as R
from gorender_gb300 import scenes
from oracle import oracle

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

NO_CLIP = gr.FLAGS_DEFAULT & ~(gr.FRUSTUM_CLIPPING | gr.BACKFACE_CULLING)


def _scene(n, flags, px=40000, w=70, h=50, seed=3, vcolor=False):
    """n triangles of up to `px` pixels around the screen's middle, both windings:
    some lie within the bound, most beyond it."""
    rng = scenes.SplitMix64(seed)
    c = rng.uniform(3 * n, -1.0, 1.0).reshape(n, 1, 3) * np.array([1.1, 1.1 * h / w, 0.3], np.float32)
    tri = c + rng.uniform(9 * n, -0.5, 0.5).reshape(n, 3, 3) * np.array([px * 1.16 / h, px * 1.16 / h, 0.05], np.float32)
    pos = np.ones((3 * n, 4), np.float32)
    pos[:, :3] = tri.reshape(-1, 3)
    vidx = np.arange(3 * n, dtype=np.int32).reshape(n, 3)
    vn = np.ones((3 * n, 4), np.float32)
    vn[:, :3] = rng.uniform(9 * n, -1.0, 1.0).reshape(3 * n, 3)
    m = scenes.MeshData(pos=pos, vidx=vidx, vnrm=vn, nidx=vidx.copy())
    m.uv = rng.uniform(6 * n, -2.0, 2.0).reshape(n, 6)
    m.tex = (np.arange(n) % 3 - 1).astype(np.int32)
    if vcolor:
        m.vcolor = rng.uniform(9 * n, 0.0, 1.0).reshape(3 * n, 3)
    tex = [scenes.random_texture(16, 16, seed=4, scale=2.0), scenes.random_texture(13, 7, seed=5, scale=1.5)]
    cam = scenes.CameraData((0.0, 0.0, 1.0), (0.0, 0.0, -1.0), (0.0, 1.0, 0.0))
    return scenes.SceneData("far", w, h, [scenes.ObjectData(m)], cam, tex, flags)


def _check(rgba, z, ref):
    assert np.array_equal(rgba, ref[0]) and np.array_equal(z.view(np.uint32), ref[1].view(np.uint32))


@pytest.mark.parametrize("extra,without,vcolor", [
    (0, 0, False), (0, gr.SHOW_TEXTURES, True), (gr.FLAT_SHADING, 0, True), (0, gr.LIGHTING, False),
    (gr.SHOW_EDGES | gr.SHOW_VERTICES, 0, False), (gr.SHOW_EDGES, gr.SHOW_FACES, False), (0, gr.SHOW_FACES, False),
    (gr.BACKFACE_CULLING, 0, True)])
def test_forms(extra, without, vcolor):
    sc = _scene(500, (NO_CLIP | extra) & ~without, px=60000 if extra & gr.SHOW_EDGES else 40000, vcolor=vcolor)
    ctx = gr.Context(0)
    try:
        up = gr.UploadedScene(ctx, sc)
        ref = oracle.draw_scene(sc, items_override=up.matrices, nthreads=4)
        rgba, z, tpf = up.render()
        assert ref[3] == 0 and tpf == ref[2] > 100
        _check(rgba, z, ref)
    finally:
        ctx.close()


def test_a_million_faces():
    sc = _scene(4001, NO_CLIP | gr.FLAT_SHADING, px=50000, w=16, h=8)
    m = sc.objects[0].mesh
    m.vidx = np.ascontiguousarray(np.resize(m.vidx, (1000003, 3)))
    m.nidx, m.uv, m.tex = m.vidx, np.resize(m.uv, (1000003, 6)), np.resize(m.tex, 1000003)
    ctx = gr.Context(0)
    try:
        up = gr.UploadedScene(ctx, sc)
        ref = oracle.draw_scene(sc, items_override=up.matrices, nthreads=8)
        rgba, z, tpf = up.render()
        assert ref[3] == 0 and tpf == ref[2] > 100000
        _check(rgba, z, ref)
    finally:
        ctx.close()


def test_batch_with_a_clipping_view():
    sc = _scene(300, NO_CLIP)
    scs = [sc, dataclasses.replace(sc, flags=sc.flags | gr.FRUSTUM_CLIPPING, width=64, height=40)]
    ctx = gr.Context(0)
    try:
        ups = [gr.UploadedScene(ctx, s) for s in scs]
        outs = [(torch.zeros((s.height, s.width, 4), dtype=torch.uint8, device="cuda"),
                 torch.zeros((s.height, s.width), device="cuda")) for s in scs]
        torch.cuda.synchronize()
        b = R.Batch(ctx, [(u.params, c.data_ptr(), d.data_ptr()) for u, (c, d) in zip(ups, outs)],
                    [(h, m[0], m[1], v) for v, u in enumerate(ups) for h, m in zip(u.mesh_handles, u.matrices)], autotune=False)
        b.run()
        b.sync()
        for s, u, (c, d) in zip(scs, ups, outs):
            ref = oracle.draw_scene(s, items_override=u.matrices, nthreads=4)
            assert ref[3] == 0 and (ref[1] > -1).any()
            _check(c.cpu().numpy(), d.cpu().numpy(), ref)
    finally:
        ctx.close()


@pytest.mark.parametrize("value", [np.nan, np.inf, 2e38])
def test_box_that_is_no_box(value):
    """One vertex that no face uses: a NaN turns every test of the box against the
    planes false, and an asynchronous frame of mostly far faces must not overflow."""
    sc = _scene(4000, gr.FLAGS_DEFAULT & ~gr.BACKFACE_CULLING, w=64, h=32)
    m = sc.objects[0].mesh
    m.pos = np.concatenate([m.pos, np.array([[value, value, value, 1.0]], np.float32)])
    ctx = gr.Context(0)
    try:
        up = gr.UploadedScene(ctx, sc)
        ref = oracle.draw_scene(sc, items_override=up.matrices, nthreads=4)
        assert ref[3] == 0 and ref[2] > 1500
        if np.isnan(value):  # the others are clipped, at most faces / 16 + 1024 of them in a first frame
            c = torch.zeros((sc.height, sc.width, 4), dtype=torch.uint8, device="cuda")
            d = torch.zeros((sc.height, sc.width), device="cuda")
            torch.cuda.synchronize()
            gr.draw_async(ctx, up.items, 1, up.params, c.data_ptr(), d.data_ptr())
            ctx.sync()
            _check(c.cpu().numpy(), d.cpu().numpy(), ref)
        rgba, z, tpf = up.render()
        assert tpf == ref[2]
        _check(rgba, z, ref)
    finally:
        ctx.close()
