"""The per-pixel kernels of the differentiable step over views of uneven shapes:
their CTAs stand in one list over all views, 32 x 8, 16 x 16 or 8 x 32 pixels a
block by the view's width, one or eight blocks a CTA by the number of pixels."""
import math

import numpy as np
import pytest

import gorender_gb300 as gr
from gorender_gb300 import renderer as R
from tests import test_gpu_diff_edges as edges

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

WIDTHS = [1, 7, 8, 9, 15, 16, 17, 31, 32, 33, 65]
HEIGHTS = [1, 3, 4, 8, 9, 15, 16, 17, 31, 32, 33, 63, 64, 65, 255, 256, 257]


def _loss(mesh, views, world, params, target):
    """The forward pass's loss, and the float32 losses of its pixels."""
    ctx = gr.Context(0)
    try:
        tex = params["tex"]
        d = R.Diff(ctx, ctx.mesh(mesh), world, views, tex_size=(0, 0) if tex is None else tex.shape[:2])
        p = [None if params[k] is None else edges._dev(params[k]) for k in ("pos", "vcol", "tex")]
        t = edges._dev(target)
        image = torch.full_like(t, 7.0)
        loss = d.forward(p[0].data_ptr(), p[1].data_ptr(), None if tex is None else p[2].data_ptr(), params["light"],
                         t.data_ptr(), image.data_ptr())
        e = image.cpu().numpy() - target
        e *= e
        return loss, ((e[:, 0] + e[:, 1]) + e[:, 2]) + e[:, 3]
    finally:
        ctx.close()


def test_line_column_and_many_single_pixels():
    """Widest by highest by number of views is 2^32 blocks and more here; the
    views' own blocks are 8 thousand."""
    sizes = [(16384, 1), (1, 16384)] + [(1, 1)] * 4095
    case = edges._case(sizes, 3, 31, seed=9)
    loss, pixels = _loss(*case)
    want = float(pixels.astype(np.float64).sum())
    assert want > 0 and abs(loss - want) <= 1e-12 * want
    edges._compare(*case)


@pytest.mark.parametrize("large", [False, True])
def test_uneven_shapes(large):
    """More views than a search takes a round; with a large view, eight blocks a CTA."""
    rng = np.random.default_rng(12)
    sizes = [(int(w), int(h)) for w in WIDTHS for h in rng.choice(HEIGHTS, 4, replace=False)]
    sizes += [(1531, 1429)] * large
    assert (sum(w * h for w, h in sizes) >= 1 << 21) == large and len(sizes) > 32
    edges._compare(*edges._case(sizes, 3, 17, seed=10))


@pytest.mark.parametrize("sizes", [[(8, 33)] * 5, [(16, 17), (8, 31)], [(17, 8), (33, 8)], [(8, 32), (32, 8), (16, 16)]])
def test_even_and_uneven_numbers_of_blocks(sizes):
    """Views of as many blocks each, in equal and in different shapes, and others."""
    edges._compare(*edges._case([(w * 3, h * 5) if w > 16 else (w, h * 9) for w, h in sizes], 4, 0, seed=11))


@pytest.mark.parametrize("size", [(131, 97), (1531, 1429)])
def test_loss_is_summed_in_64_bits(size):
    """Losses in the pixels of one warp only (8 x 4, or eight such blocks one below
    the other), one large among small ones, whose sum a pair of float32 rounds to
    about 46 bits.  Nothing but zeros is added to the warp's own value, which rounds
    three times."""
    mesh, views, world, params, _ = edges._case([size], 3, 0, seed=13)
    w, h = size
    rows = [y for y in range(0, 64 if w * h >= 1 << 21 else 8) if y % 8 < 4]
    at = np.array([y * w + x for y in rows for x in range(8)])
    rng = np.random.default_rng(14)
    ctx = gr.Context(0)
    try:
        d = R.Diff(ctx, ctx.mesh(mesh), world, views, tex_size=(0, 0))
        pos, vcol = edges._dev(params["pos"]), edges._dev(params["vcol"])
        zero = torch.zeros((w * h, 4), device="cuda")
        image = torch.empty_like(zero)
        forward = lambda t, i: d.forward(pos.data_ptr(), vcol.data_ptr(), None, params["light"], t.data_ptr(), i.data_ptr())
        forward(zero, image)
        for _ in range(40):
            target = image.cpu().numpy().copy()
            add = np.where(rng.random(len(at)) < 1 / 16, 1.0, 1.5e-4 * (0.5 + rng.random(len(at))))
            target[at, 0] += add.astype(np.float32)
            loss = forward(edges._dev(target), torch.empty_like(zero))
            e = (image.cpu().numpy() - target)[at, 0]
            want = math.fsum((e * e).astype(np.float64).tolist())
            assert want > 0 and abs(loss - want) <= 3 * 2.0 ** -53 * want
    finally:
        ctx.close()
