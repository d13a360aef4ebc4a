"""The persistent token-block GEMM where its tiles and its float32 epilogue can go wrong: every tile width with ragged last tiles, tiles
that lie in two blocks of the activation image, products that are ties between two floats, scales at the ends of their range, and
the widest rows whose sums the float32 epilogue takes.  All outputs are compared bit for bit with integer sums and float64."""
import numpy as np
import pytest

import loom_b200
from loom_b200 import cabi
from oracle import oracle as orc
from refkit import np_unpack

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = loom_b200.Context(0)
    yield c
    c.close()


def check(ctx, words, scale, x, rows, cols, act=cabi.ACT_LINEAR, residual=None, pre=False):
    tokens = len(x)
    w = ctx.upload_ternary(words, rows, cols, scale)
    dx, dout = ctx.to_device(x), ctx.alloc(tokens * rows * 4)
    dr = ctx.to_device(residual) if residual is not None else None
    ctx.ternary_gemm(w, tokens, dx, out=dout, residual=dr, act=act)
    out = ctx.download(dout, (tokens, rows), np.float32)
    q, amax = orc.quantize_rows_f32(x)
    # float64 sums of integers below 2^53 are exact
    acc = q.astype(np.float64) @ np_unpack(words, rows, cols).astype(np.float64).T
    os_ = np.float64(np.float32(scale)) * amax.astype(np.float64) / 127.0
    os_[os_ == 0] = 1.0
    with np.errstate(over="ignore"):
        f = (acc * os_[:, None]).astype(np.float32)
    if act == cabi.ACT_RELU2:
        f = np.where(f < 0, np.float32(0), f * f)
    if residual is not None:
        f = f + residual
    assert (out.view(np.uint32) == f.view(np.uint32)).all()
    for p in (dx, dout, dr):
        if p:
            ctx.free(p)


def matrix(rng, rows, cols):
    m = orc.Matrix.from_f32((rng.standard_normal(rows * cols) * 0.02).astype(np.float32), rows, cols)
    return m.words, float(m.scale)


# the rule's choice (0) and both widths an option can ask for; 47 to 700 tokens make it choose 48 to 256
@pytest.mark.parametrize("tile", [0, 128, 256])
@pytest.mark.parametrize("rows,cols,tokens", [(2560, 300, 1024), (2560, 129, 640), (4096, 256, 700), (640, 640, 47), (129, 128, 511), (6912, 128, 257), (20000, 64, 333)])
def test_tile_widths(ctx, rows, cols, tokens, tile):
    rng = np.random.default_rng(rows + tokens)
    ctx.set_option("gemm_tile", tile)
    try:
        check(ctx, *matrix(rng, rows, cols), rng.standard_normal((tokens, cols)).astype(np.float32), rows, cols, residual=rng.standard_normal((tokens, rows)).astype(np.float32))
    finally:
        ctx.set_option("gemm_tile", 0)


def test_products_between_two_floats(ctx):
    # scale 127 makes the output scale the token's largest value itself; 24 odd bits of it times a small sum are often half way between floats
    rng = np.random.default_rng(1)
    rows, cols, tokens = 256, 32, 300
    x = np.zeros((tokens, cols), np.float32)
    odd = (0x3f800001 + 2 * rng.integers(0, 1 << 22, tokens)).astype(np.uint32).view(np.float32)
    x[:, 0] = odd
    x[:, 1:5] = (odd[:, None] * rng.integers(-6, 7, (tokens, 4)) / 127).astype(np.float32)
    words, _ = matrix(rng, rows, cols)
    check(ctx, words, 127.0, x, rows, cols, act=cabi.ACT_RELU2)
    check(ctx, words, 127.0, x, rows, cols)


@pytest.mark.parametrize("scale", [-0.5, 1e-38, 1e-25, 1e-12, 1e15, 1e30, 3e38])
@pytest.mark.parametrize("spread", [1e-7, 1.0, 1e6])
def test_scales(ctx, scale, spread):
    rng = np.random.default_rng(2)
    rows, cols, tokens = 200, 100, 65
    words, _ = matrix(rng, rows, cols)
    check(ctx, words, scale, (rng.standard_normal((tokens, cols)) * spread).astype(np.float32), rows, cols)


@pytest.mark.parametrize("cols", [32512, 32640, 32641, 32768])
def test_widest_rows(ctx, cols):
    # every code 2 and every value the largest: the sum is +-127 * cols
    rng = np.random.default_rng(cols)
    rows, tokens = 70, 40
    words = np.full((rows, (cols + 15) // 16), 0xAAAAAAAA, np.uint32)
    words[rows // 2:] = rng.integers(0, 2, words[rows // 2:].shape).astype(np.uint32) * 0x55555555 + 0x00000000
    x = np.ones((tokens, cols), np.float32)
    x[1::2] *= -1
    x[4:] = rng.standard_normal((tokens - 4, cols))
    check(ctx, words, 0.0123, x, rows, cols)
