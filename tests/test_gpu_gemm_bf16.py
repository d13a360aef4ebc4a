"""The bf16 token-block product by itself, column by column.  Rows and weights are small whole numbers over 32, so that every float32 sum
is exact in any order: outputs without a function must be the exact sums (rounded once where they are stored as bf16), the others
within one rounding to bf16 and the function's few float32 roundings.  Sizes make the tiles 48 to 256 columns wide, one to many waves of
them, with ragged last tiles, slices and tokens."""
import numpy as np
import pytest
import torch

import loom_b200
from harness import lib
from loom_b200 import cabi

pytestmark = pytest.mark.gpu
F32, RESID, GELU, GLU, IMG, HEADS, SILU = 0, 1, 2, 3, 4, 5, 7
SHAPES = [(1, 16, 64), (5, 130, 100), (47, 48, 70), (100, 2560, 6912), (33, 300, 1000), (129, 1000, 520), (700, 2000, 192), (2100, 2570, 128), (640, 20000, 64), (333, 7696, 256)]


@pytest.fixture(scope="module")
def ctx():
    c = loom_b200.Context(0)
    yield c
    c.close()


def matrix(ctx, a):
    return cabi.Matrix(ctx, *a.shape).put(np.ascontiguousarray(a, np.float32))


def rows_of_image(raw, rows, cols, slices):
    """bf16 rows of an image [row block][slice][row / 8][chunk][row % 8][8] (or of per-head blocks, a head for a slice), as float64"""
    a = (raw.astype(np.uint32) << 16).view(np.float32).reshape(-1, slices, 16, raw.size // (-(-rows // 128) * slices * 1024), 8, 8)
    return a.transpose(0, 2, 4, 1, 3, 5).reshape(a.shape[0] * 128, slices, -1)[:rows].astype(np.float64)


def product(ctx, epi, x, w, w2=None, out=None, ldo=0, img=None, slices=0, heads=0, hd=0, mult=1.0, res=1.0, limit=0.0):
    ctx._check(lib().t_gemm_bf16(ctx.h, epi, x.h, w.h, w2.h if w2 else None, x.rows, out, ldo, img, slices, heads, hd, mult, res, limit))


def bf16(a):
    return torch.from_numpy(a).to(torch.bfloat16).to(torch.float64).numpy()


@pytest.mark.parametrize("tokens,rows,cols", SHAPES)
def test_every_column(ctx, tokens, rows, cols):
    rng = np.random.default_rng(rows + tokens)
    xs, ws, us = (rng.integers(-3, 4, s).astype(np.float32) for s in ((tokens, cols), (rows, cols), (rows, cols)))
    xs /= 32
    x, w, u = matrix(ctx, xs), matrix(ctx, ws), matrix(ctx, us)
    sums, ups = (xs.astype(np.float64) @ m.T.astype(np.float64) for m in (ws, us))
    ldo = -(-rows // 8) * 8
    first = rng.integers(-50, 50, (tokens, ldo)).astype(np.float32)
    out = ctx.to_device(first)
    for epi, want in ((RESID, sums * 0.5 + 2.0 * first[:, :rows]), (F32, sums)):
        product(ctx, epi, x, w, out=out, ldo=ldo, mult=0.5, res=2.0)
        got = ctx.download(out, (tokens, ldo), np.float32)
        assert (got[:, :rows] == want).all()
        assert epi == RESID or (got[:, rows:] == 0).all()
    slices = -(-rows // 64)
    words = -(-tokens // 128) * slices * 8192
    img = ctx.to_device(np.full(words, 0x7FC0, np.uint16))
    z = np.clip(sums, None, 7.0)
    half_erf = 0.5 * sums * torch.special.erfc(torch.from_numpy(-sums / np.sqrt(2.0))).numpy()
    for epi, second, want in ((IMG, None, sums), (GELU, None, half_erf), (GLU, u, z / (1 + np.exp(-1.702 * z)) * (np.clip(ups, -7.0, 7.0) + 1)),
                              (SILU, u, sums / (1 + np.exp(-sums)) * ups)):
        product(ctx, epi, x, w, second, img=img, slices=slices, limit=7.0)
        got = rows_of_image(ctx.download(img, (words,), np.uint16), tokens, rows, slices).reshape(tokens, -1)
        assert (got[:, rows:] == 0).all()
        got = got[:, :rows]
        if epi == IMG:
            assert (got == bf16(want.astype(np.float32))).all()
        else:  # half a unit of bf16 (8 bits of significand), a few roundings of float32 (of the sum 1 + erf, where it is small)
            assert (np.abs(got - want) <= (2.0 ** -8 + 2.0 ** -18) * np.abs(want) + 2.0 ** -22 * np.abs(sums) * (1 + np.abs(ups) * (epi != GELU))).all()
    for hd in [d for d in (8, 16, 40) if rows % d == 0]:
        heads, chunks = rows // hd, hd // 8
        words = -(-tokens // 128) * heads * chunks * 1024
        blocks = ctx.to_device(np.full(words, 0x7FC0, np.uint16))
        product(ctx, HEADS, x, w, img=blocks, heads=heads, hd=hd)
        got = rows_of_image(ctx.download(blocks, (words,), np.uint16), tokens, rows, heads)
        assert (got.reshape(tokens, rows) == bf16(sums.astype(np.float32))).all()
        ctx.free(blocks)
    for p in (out, img):
        ctx.free(p)
    for m in (x, w, u):
        m.free()


@pytest.mark.parametrize("rows,cols", [(2560, 6912), (640, 2560), (7696, 2560), (300, 4096)])
def test_a_token_has_its_bits_in_any_block(ctx, rows, cols):
    """One accumulator takes all of K: a token's sums are the same bits whether few tokens are in its block or many."""
    rng = np.random.default_rng(rows)
    xs, w = rng.standard_normal((2100, cols)).astype(np.float32), matrix(ctx, rng.standard_normal((rows, cols)).astype(np.float32) * cols ** -0.5)
    ldo = -(-rows // 8) * 8
    got = {}
    for n in (2100, 1030, 128, 100, 3):
        x, out = matrix(ctx, xs[:n]), ctx.alloc(n * ldo * 4)
        product(ctx, F32, x, w, out=out, ldo=ldo)
        got[n] = ctx.download(out, (n, ldo), np.float32)
        ctx.free(out)
        x.free()
        assert np.array_equal(got[n].view(np.uint32), got[2100][:n].view(np.uint32))
    w.free()
