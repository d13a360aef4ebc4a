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


# rows of blocks of many tokens are quantized behind bulk copies, a thread per sixteen columns: 256, 512 and 1024 threads, ragged last
# chunks, rows that bulk copies cannot take (columns not a multiple of four) or that are too wide
@pytest.mark.parametrize("cols,tokens", [(4, 296), (20, 297), (102, 300), (252, 513), (4096, 296), (4100, 300), (8192, 297), (8196, 301), (16384, 296), (16388, 299)])
def test_quantized_rows_of_many_tokens(ctx, cols, tokens):
    rng = np.random.default_rng(cols)
    x = rng.standard_normal((tokens, cols)).astype(np.float32)
    x[5] = 0
    x[7, 0] = 1e30
    # values whose codes lie half way between two integers, from either side
    x[9:40] = ((rng.integers(-127, 127, (31, cols)) + 0.5) / 127).astype(np.float32)
    x[9:40, 0] = 1
    check(ctx, *matrix(rng, 64, cols), x, 64, cols)


@pytest.mark.parametrize("heads,hd,inter", [(4, 16, 320), (3, 16, 4400), (2, 24, 8400), (20, 16, 17000)])
def test_normed_rows_of_many_tokens(heads, hd, inter):
    # prompts of more than two tokens an SM: block norm, inner norm of float64 and of float32 rows; logits as in test_gpu_attention_prompt.py
    rng = np.random.default_rng(inter)
    c = loom_b200.Context(0)
    H, V, L, msl = heads * hd, 64, 2, 512
    shapes = ((H, H), (hd, H), (hd, H), (H, H), (inter, H), (inter, H), (H, inter))
    gdec = cabi.Decoder(c, L, H, heads, 1, hd, inter, V, 1e-5, 500000.0, cabi.ACT_SILU, msl)
    odec = orc.Decoder(L, H, heads, 1, hd, inter, V, 1e-5, 500000.0, orc.ACT_SILU, msl)
    try:
        for b in range(L):
            packed = [orc.pack_f32((rng.standard_normal(r * k) * 0.02).astype(np.float32), r, k) for r, k in shapes]
            gdec.set_block(b, [c.upload_ternary(p[0], r, k, p[1]) for p, (r, k) in zip(packed, shapes)])
            odec.set_block_packed(b, [p[0] for p in packed], [p[1] for p in packed])
        emb = (rng.standard_normal((V, H)) * 0.02).astype(np.float32)
        gdec.set_embeddings(c.to_device(emb))
        odec.set_embeddings(emb)
        tok = rng.integers(0, V, 301).astype(np.int32)
        got, want = gdec.forward(tok), odec.forward(tok, threads=min(16, orc.host_threads()))
        assert np.max(np.abs(got - want)) <= 1e-6 * max(1.0, float(np.max(np.abs(want))))
    finally:
        gdec.close()
        c.close()


@pytest.mark.parametrize("cols", [64, 1000, 16384])
def test_rows_that_are_not_numbers(ctx, cols):
    """Infinities, NaN, the largest and the smallest numbers, zeros of both signs: the float quantizer and the rows that bulk copies bring give
    what the former quantizer gives, codes, largest values and sums."""
    rng = np.random.default_rng(cols)
    rows, tokens = 70, 300
    x = rng.standard_normal((tokens, cols)).astype(np.float32)
    special = np.array([np.inf, -np.inf, np.nan, 3.4e38, -3.4e38, 1e-45, -1e-45, 0.0, -0.0, 1e-5, 9.9e-6], np.float32)
    for i, v in enumerate(special):
        x[2 * i, rng.integers(0, cols)] = v
        x[2 * i + 1] = v
    x[40] *= 1e-30
    x[41, ::2] = np.nan
    words, scale = matrix(rng, rows, cols)
    w, dx = ctx.upload_ternary(words, rows, cols, scale), ctx.to_device(x)
    got = []
    for regs in (0, 1):
        ctx.set_option("quant_regs", regs)
        try:
            out, acc, amax = ctx.alloc(tokens * rows * 4), ctx.alloc(tokens * rows * 4), ctx.alloc(tokens * 4)
            ctx.ternary_gemm(w, tokens, dx, out=out, acc_out=acc, amax_out=amax)
            plain = ctx.alloc(tokens * rows * 4)
            ctx.ternary_gemm(w, tokens, dx, out=plain)  # (without raw sums: the float epilogue)
            got.append([ctx.download(p, s, np.uint32) for p, s in ((out, (tokens, rows)), (acc, (tokens, rows)), (amax, (tokens,)), (plain, (tokens, rows)))])
        finally:
            ctx.set_option("quant_regs", 1)
    for a, b in zip(*got):
        assert (a == b).all()
    f, g = (a.view(np.float32) for a in (got[1][0], got[1][3]))
    assert ((f == g) | (np.isnan(f) & np.isnan(g))).all()
    finite = np.isfinite(x).all(1)
    q, amax = orc.quantize_rows_f32(x[finite])
    assert (got[1][2][finite].view(np.float32) == amax).all()
    assert (got[1][1][finite].view(np.int32) == (q.astype(np.float64) @ np_unpack(words, rows, cols).astype(np.float64).T)).all()
