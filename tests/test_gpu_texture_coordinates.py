"""Texture coordinates at the line between the 32-bit and the general
conversion, bit for bit against the oracle: UVs and scales whose products pass
2^31 either way, NaN and infinities, for mask and modulo textures."""
import numpy as np
import pytest

import gorender_gb300 as gr
from gorender_gb300 import scenes
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side", [(16, 16), (23, 17)])
@pytest.mark.parametrize("scale", [1.0, 1e6, 2.0 ** 27, 1e30])
def test_texture_coordinates(side, scale):
    m = scenes.heightfield(24, seed=3)
    rng = scenes.SplitMix64(5)
    m.uv = rng.uniform(6 * m.nf, -3.0, 3.0).reshape(m.nf, 6)
    m.uv[::17, 2] = np.nan
    m.uv[5::17, 3] = np.inf
    m.uv[9::17, 4] = -np.inf
    m.tex = np.zeros(m.nf, np.int32)
    tex = scenes.random_texture(*side, seed=2, scale=scale)
    cam = scenes.CameraData((0.3, 0.9, 2.5), (0.0, -0.4, -1.0), (0.0, 1.0, 0.0))
    sc = scenes.SceneData("uv", 201, 103, [scenes.ObjectData(m)], cam, [tex], gr.FLAGS_DEFAULT | gr.FLAT_SHADING)
    ctx = gr.Context(0)
    try:
        up = gr.UploadedScene(ctx, sc)
        rgba, z, tpf = up.render()
        ref = oracle.draw_scene(sc, items_override=up.matrices, nthreads=4)
        assert ref[3] == 0 and tpf == ref[2] and (ref[1] > -1).mean() > 0.2
        assert np.array_equal(rgba, ref[0]) and np.array_equal(z.view(np.uint32), ref[1].view(np.uint32))
    finally:
        ctx.close()
