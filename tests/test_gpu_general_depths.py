"""Triangles that the raster's exact division does not take, bit for bit against
the oracle: narrow ones whose W's are out of its range walk the units with general
divisions, alone and in tables with others, and those with int64 edges share their
blocks among the warps, from one block each to whole tiles."""
import numpy as np
import pytest

import gorender_gb300 as gr
from gorender_gb300 import _native as N
from gorender_gb300 import scenes
from oracle import oracle

pytestmark = pytest.mark.gpu

FLAGS = (gr.FLAGS_DEFAULT | gr.FLAT_SHADING) & ~(gr.BACKFACE_CULLING | gr.FRUSTUM_CLIPPING)


def _mesh(size, n, seed, h, spread=1.0):
    """n triangles of about `size` pixels around z = -1, a fifth of them copies."""
    rng = scenes.SplitMix64(seed)
    c = rng.uniform(3 * n, -1.0, 1.0).reshape(n, 1, 3) * np.array([1.1 * spread, 0.6 * spread, 0.3], np.float32)
    tri = c + rng.uniform(9 * n, -0.5, 0.5).reshape(n, 3, 3) * np.array([size * 1.16 / h, size * 1.16 / h, 0.2], np.float32)
    tri[..., 2] -= 1.0
    copies = np.arange(0, n, 5)[1:]
    tri[copies] = tri[copies - 1]
    pos = np.ones((3 * n, 4), np.float32)
    pos[:, :3] = tri.reshape(-1, 3)
    return scenes.MeshData(pos=pos, vidx=np.arange(3 * n, dtype=np.int32).reshape(n, 3))


def _check(objects, tile, w=130, h=70):
    cam = scenes.CameraData((0.0, 0.0, 0.0), (0.0, 0.0, -1.0), (0.0, 1.0, 0.0))
    sc = scenes.SceneData("depths", w, h, objects, cam, [], FLAGS)
    ctx = gr.Context(0)
    try:
        ctx.set_tuning(tile, 0)
        for cost in (1 << 20, 64):  # one slice a tile, and as many as there can be
            N.check(N.lib().gr_context_set_raster(ctx.handle, cost, 0))
            up = gr.UploadedScene(ctx, sc)
            ref = oracle.draw_scene(sc, items_override=up.matrices, nthreads=4)
            rgba, z, tpf = up.render()
            assert ref[3] == 0 and tpf == ref[2]
            assert np.array_equal(rgba, ref[0])
            assert np.array_equal(z.view(np.uint32), ref[1].view(np.uint32))
            assert (z > -1).any()
    finally:
        ctx.close()
    return z


@pytest.mark.parametrize("tile", [32, 16])
@pytest.mark.parametrize("size,n", [(2, 3000), (8, 900), (33, 300), (200, 40)])
@pytest.mark.parametrize("scale", [2.0 ** -62, 2.0 ** 62])
def test_w_out_of_range(tile, size, n, scale):
    """All triangles, or one object of three, whose entries lie in tables with others'."""
    s = (scale,) * 3
    far = scenes.ObjectData(_mesh(size, n, 3, 70), scale=s)
    _check([far], tile)
    near = [scenes.ObjectData(_mesh(size, n, k, 70)) for k in (4, 5)]
    z = _check([near[0], far, near[1]], tile)
    assert (np.abs(z) < 100).any()


@pytest.mark.parametrize("tile", [32, 16])
@pytest.mark.parametrize("small", [0, 9])
def test_int64_edges(tile, small):
    """Triangles over the whole screen and beyond it, slivers whose boxes clip to
    a row or a column of a few tiles, and narrow ones among them."""
    big = _mesh(60000, 300, 6, 70)
    long = _mesh(3, 600, 7, 70)
    p = long.pos.reshape(-1, 3, 4)
    p[::2, 0, 0] += np.float32(400.0)  # one corner far to the side: boxes a few rows high
    p[1::2, 0, 1] += np.float32(400.0)
    objects = [scenes.ObjectData(long), scenes.ObjectData(big)]
    if small:
        objects.insert(1, scenes.ObjectData(_mesh(small, 500, 8, 70)))
        objects.append(scenes.ObjectData(_mesh(small, 500, 9, 70), scale=(2.0 ** -62,) * 3))
    _check(objects, tile)
