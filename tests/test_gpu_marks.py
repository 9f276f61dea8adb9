"""k_overlay's tasks, a part of 32 triangles a warp: frames that ask for some of the
parts only, numbers of triangles around a warp's, and batches whose views ask for
different ones, bit for bit against the oracle."""
import numpy as np
import pytest

import gorender_gb300 as gr
from gorender_gb300 import renderer as R
from gorender_gb300 import scenes
from oracle import oracle

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

EDGES, VERTICES, FACES = gr.SHOW_EDGES, gr.SHOW_VERTICES, gr.SHOW_FACES
BASE = (gr.FLAGS_DEFAULT | gr.FLAT_SHADING) & ~(gr.BACKFACE_CULLING | FACES)


def _scene(n, flags, seed=3, w=130, h=70):
    rng = scenes.SplitMix64(seed)
    c = rng.uniform(3 * n, -1.0, 1.0).reshape(n, 1, 3) * np.array([1.1, 0.6, 0.3], np.float32)
    size = np.where(np.arange(n) % 3 == 0, 40.0, 2.0).reshape(n, 1, 1)  # two thirds cover hardly a pixel
    tri = c + rng.uniform(9 * n, -0.5, 0.5).reshape(n, 3, 3) * size * 1.16 / h
    pos = np.ones((3 * n, 4), np.float32)
    pos[:, :3] = tri.reshape(-1, 3)
    m = scenes.MeshData(pos=pos, vidx=np.arange(3 * n, dtype=np.int32).reshape(n, 3))
    cam = scenes.CameraData((0.0, 0.0, 1.0), (0.0, 0.0, -1.0), (0.0, 1.0, 0.0))
    return scenes.SceneData("marks", w, h, [scenes.ObjectData(m)], cam, [], flags)


@pytest.mark.parametrize("n", [1, 31, 33, 900])
@pytest.mark.parametrize("marks", [EDGES, VERTICES, EDGES | FACES, VERTICES | FACES, EDGES | VERTICES, EDGES | VERTICES | FACES])
def test_parts(n, marks):
    sc = _scene(n, BASE | marks)
    ctx = gr.Context(0)
    try:
        up = gr.UploadedScene(ctx, sc)
        ref = oracle.draw_scene(sc, items_override=up.matrices, nthreads=4)
        rgba, z, tpf = up.render()
        assert ref[3] == 0 and tpf == ref[2]
        assert np.array_equal(rgba, ref[0]) and np.array_equal(z.view(np.uint32), ref[1].view(np.uint32))
    finally:
        ctx.close()


@pytest.mark.parametrize("views", [[EDGES, VERTICES | FACES, FACES], [VERTICES, FACES, VERTICES | FACES],
                                   [EDGES | FACES, FACES, EDGES]])
def test_batch_of_different_marks(views):
    scs = [_scene(300, BASE | f, seed=5) for f in views]
    ctx = gr.Context(0)
    try:
        up = gr.UploadedScene(ctx, scs[0])
        outs = [(torch.zeros((s.height, s.width, 4), dtype=torch.uint8, device="cuda"),
                 torch.zeros((s.height, s.width), device="cuda")) for s in scs]
        torch.cuda.synchronize()
        b = R.Batch(ctx, [(R.make_params(s.width, s.height, s.flags), c.data_ptr(), d.data_ptr()) for s, (c, d) in zip(scs, outs)],
                    [(h, m[0], m[1], v) for v in range(len(scs)) for h, m in zip(up.mesh_handles, up.matrices)], autotune=False)
        b.run()
        b.sync()
        for s, (c, d) in zip(scs, outs):
            ref = oracle.draw_scene(s, items_override=up.matrices, nthreads=4)
            assert ref[3] == 0
            assert np.array_equal(c.cpu().numpy(), ref[0])
            assert np.array_equal(d.cpu().numpy().view(np.uint32), ref[1].view(np.uint32))
    finally:
        ctx.close()
