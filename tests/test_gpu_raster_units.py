"""The raster's unit walk at the sizes where it can go wrong, bit for bit
against the oracle: bins of one entry, of a whole batch and of one more (256
entries at 32 x 32 tiles, 64 at 16 x 16), tiles of tiny triangles (at most 3 x 3
pixels, points and slivers among them), boxes one pixel either side of a unit
(8 pixels) and of a tile, slices without entries, W's beyond the range of
the exact division (the general path), and their mixtures."""
import numpy as np
import pytest

import gorender_gb300 as gr
from gorender_gb300 import _native as N
from gorender_gb300 import renderer as R
from gorender_gb300 import scenes
from oracle import oracle

pytestmark = pytest.mark.gpu

FLAGS = (gr.FLAGS_DEFAULT | gr.FLAT_SHADING) & ~gr.BACKFACE_CULLING


def _scene(size, n, seed, w=130, h=70, far=1.0):
    """n triangles of about `size` pixels over the frame, both windings, a
    fifth of them copies (depth ties); far scales the scene, and with it W."""
    rng = scenes.SplitMix64(seed)
    c = rng.uniform(3 * n, -1.0, 1.0).reshape(n, 1, 3) * np.array([1.1, 0.6, 0.3], np.float32)
    tri = c + rng.uniform(9 * n, -0.5, 0.5).reshape(n, 3, 3) * np.float32(size * 1.16 / h)
    copies = np.arange(0, n, 5)[1:]
    tri[copies] = tri[copies - 1]
    pos = np.ones((3 * n, 4), np.float32)
    pos[:, :3] = tri.reshape(-1, 3) * np.float32(far)
    m = scenes.MeshData(pos=pos, vidx=np.arange(3 * n, dtype=np.int32).reshape(n, 3))
    cam = scenes.CameraData((0.0, 0.0, far), (0.0, 0.0, -1.0), (0.0, 1.0, 0.0))
    return scenes.SceneData("units", w, h, [scenes.ObjectData(m)], cam, [], FLAGS)


@pytest.mark.parametrize("tile", [32, 16])
@pytest.mark.parametrize("size,n", [(1, 3000), (2, 6000), (3, 2500), (7, 900), (9, 700), (30, 257), (34, 64), (80, 65),
                                    (400, 1), (400, 9), (400, 300)])
def test_units(tile, size, n):
    ctx = gr.Context(0)
    try:
        ctx.set_tuning(tile, 0)
        sc = _scene(size, n, seed=3 + 10 * size + n)
        for cost in (1 << 20, 64):  # one slice a tile, and as many as there can be
            N.check(N.lib().gr_context_set_raster(ctx.handle, cost, 0))
            up = gr.UploadedScene(ctx, sc)
            rgba, z, tpf = up.render()
            ref = oracle.draw_scene(sc, items_override=up.matrices, nthreads=4)
            assert ref[3] == 0 and tpf == ref[2]
            assert np.array_equal(rgba, ref[0])
            assert np.array_equal(z.view(np.uint32), ref[1].view(np.uint32))
            assert (z > -1).any()
    finally:
        ctx.close()


@pytest.mark.parametrize("far", [2.0 ** -58, 2.0 ** -63])
def test_units_and_general_path_by_w(far):
    """W's of about 2^-58 take the units, of 2^-63 the general path; clipping
    is off (the planes stand at W's of 1) and the depths are huge."""
    ctx = gr.Context(0)
    try:
        sc = _scene(20, 200, seed=7, far=far)
        sc.flags &= ~gr.FRUSTUM_CLIPPING
        up = gr.UploadedScene(ctx, sc)
        rgba, z, tpf = up.render()
        ref = oracle.draw_scene(sc, items_override=up.matrices, nthreads=4)
        assert ref[3] == 0 and tpf == ref[2]
        assert np.array_equal(rgba, ref[0]) and np.array_equal(z.view(np.uint32), ref[1].view(np.uint32))
        assert (z > -1).any()
    finally:
        ctx.close()


@pytest.mark.parametrize("tile", [32, 16])
def test_huge_triangles(tile):
    """Triangles over more than 256 tiles, which k_plan bins: whole and clipped
    (the camera among them), more of them than its list holds (1024), alone and
    in a batch with a view of few tiles."""
    torch = pytest.importorskip("torch")

    ctx = gr.Context(0)
    try:
        ctx.set_tuning(tile, 0)
        scs = [_scene(1500, 30, seed=5, w=1101, h=603), _scene(3000, 6, seed=6, w=64, h=40),
               _scene(1500, 2600, seed=8, w=640, h=420)]
        for sc in scs[:2]:  # corners behind the camera too
            sc.objects[0].mesh.pos[::4, 2] += np.float32(1.5)
        views, entries, outs = [], [], []
        for v, sc in enumerate(scs):
            up = gr.UploadedScene(ctx, sc)
            ref = oracle.draw_scene(sc, items_override=up.matrices, nthreads=4)
            rgba, z, tpf = up.render()
            assert ref[3] == 0 and tpf == ref[2] and (ref[1] > -1).any()
            assert np.array_equal(rgba, ref[0]) and np.array_equal(z.view(np.uint32), ref[1].view(np.uint32))
            c = torch.zeros((sc.height, sc.width, 4), dtype=torch.uint8, device="cuda")
            d = torch.zeros((sc.height, sc.width), dtype=torch.float32, device="cuda")
            outs.append((up, ref, c, d))
            views.append((up.params, c.data_ptr(), d.data_ptr()))
            entries += [(h, m[0], m[1], v) for h, m in zip(up.mesh_handles, up.matrices)]
        torch.cuda.synchronize()
        b = R.Batch(ctx, views, entries, autotune=False)
        b.run()
        b.sync()
        for _, ref, c, d in outs:
            assert np.array_equal(c.cpu().numpy(), ref[0])
            assert np.array_equal(d.cpu().numpy().view(np.uint32), ref[1].view(np.uint32))
    finally:
        ctx.close()


def test_far_faces_of_unclipped_views():
    """Without clipping most faces may have corners beyond the narrow bound:
    k_clip sets them up whole, and an asynchronous frame of them fits the
    buffers that its size gets at once."""
    torch = pytest.importorskip("torch")
    sc = _scene(60000, 1500, seed=11, w=70, h=50)
    sc.flags &= ~gr.FRUSTUM_CLIPPING
    ref = oracle.draw_scene(sc, nthreads=4)
    assert ref[3] == 0 and (ref[1] > -1).any()
    ctx = gr.Context(0)
    try:
        up = gr.UploadedScene(ctx, sc)
        c = torch.zeros((sc.height, sc.width, 4), dtype=torch.uint8, device="cuda")
        d = torch.zeros((sc.height, sc.width), dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
        gr.draw_async(ctx, up.items, 1, up.params, c.data_ptr(), d.data_ptr())
        ctx.sync()
        assert np.array_equal(c.cpu().numpy(), ref[0])
        assert np.array_equal(d.cpu().numpy().view(np.uint32), ref[1].view(np.uint32))
        assert up.draw() == ref[2]
    finally:
        ctx.close()


@pytest.mark.parametrize("flags", [0, gr.SHOW_EDGES, gr.SHOW_VERTICES])
@pytest.mark.parametrize("faces", [True, False])
def test_small_triangles_with_marks_and_without_faces(flags, faces):
    """Triangles that cover no pixel count in TPF and leave their marks."""
    sc = _scene(2, 3000, seed=23)
    sc.flags = (sc.flags | flags) & ~(0 if faces else gr.SHOW_FACES)
    ctx = gr.Context(0)
    try:
        up = gr.UploadedScene(ctx, sc)
        rgba, z, tpf = up.render()
        ref = oracle.draw_scene(sc, items_override=up.matrices, nthreads=4)
        assert ref[3] == 0 and tpf == ref[2] > 1000
        assert np.array_equal(rgba, ref[0]) and np.array_equal(z.view(np.uint32), ref[1].view(np.uint32))
    finally:
        ctx.close()


@pytest.mark.parametrize("faces", [1000001, 2000003, 4000000, 4002055])
def test_faces_a_thread(faces):
    """2, 4 and 8 faces a thread in k_cull, with a last CTA that is not full."""
    sc = _scene(2, 4001, seed=37)
    m = sc.objects[0].mesh
    m.vidx = np.ascontiguousarray(np.resize(m.vidx, (faces, 3)))
    ctx = gr.Context(0)
    try:
        up = gr.UploadedScene(ctx, sc)
        rgba, z, tpf = up.render()
        ref = oracle.draw_scene(sc, items_override=up.matrices, nthreads=8)
        assert ref[3] == 0 and tpf == ref[2] > faces // 2
        assert np.array_equal(rgba, ref[0]) and np.array_equal(z.view(np.uint32), ref[1].view(np.uint32))
    finally:
        ctx.close()


@pytest.mark.parametrize("strength", [1.0, -3.0, 300.0, 65534.9, 65535.1, 1e9, 1e38, np.inf, np.nan])
def test_intensities(strength):
    """Colours times intensities below zero, around 2^15 (products of 2^23 and
    more are converted the general way), beyond whole numbers, infinite and NaN,
    shaded by k_resolve and in place."""
    torch = pytest.importorskip("torch")
    sc = _scene(9, 900, seed=41)
    light = np.array([0.3, 0.2, 1.0], np.float32) * np.float32(strength)
    ctx = gr.Context(0)
    try:
        up = gr.UploadedScene(ctx, sc)
        for k in range(3):
            up.params.light[k] = float(light[k])
        ref = oracle.draw_scene(sc, items_override=up.matrices, light=light, nthreads=4)
        rgba, z, tpf = up.render()
        assert ref[3] == 0 and tpf == ref[2] and len(np.unique(ref[0][..., 0])) > 1
        assert np.array_equal(rgba, ref[0]) and np.array_equal(z.view(np.uint32), ref[1].view(np.uint32))
        outs = [(torch.zeros((sc.height, sc.width, 4), dtype=torch.uint8, device="cuda"),
                 torch.zeros((sc.height, sc.width), dtype=torch.float32, device="cuda")) for _ in range(2)]
        torch.cuda.synchronize()
        b = R.Batch(ctx, [(up.params, c.data_ptr(), d.data_ptr()) for c, d in outs],
                    [(h, m[0], m[1], v) for v in range(2) for h, m in zip(up.mesh_handles, up.matrices)], autotune=False)
        b.run()
        b.sync()
        for c, d in outs:
            assert np.array_equal(c.cpu().numpy(), ref[0])
    finally:
        ctx.close()
