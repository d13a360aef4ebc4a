"""Ternary products of 3 to 24 tokens per pass: one to three MMA columns of tokens, one to eight CTAs to a cluster, ragged last strips and
columns, more rows than one wave of CTAs holds, rows too wide for the pass, products so small that the one-token kernel keeps them.  Sums, outputs and codes are compared bit for bit."""
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


# (cols: 1 to 256 blocks of 128 columns)
SHAPES = [(16, 128), (40, 100), (1024, 128), (1025, 128), (33, 1000), (2560, 6912), (6912, 2560), (300, 14336), (5, 32768), (70, 32769), (140000, 64), (130, 511)]


@pytest.mark.parametrize("rows,cols", SHAPES)
@pytest.mark.parametrize("tokens", [3, 5, 6, 8, 9, 16, 23, 24, 25, 29])
def test_linear(ctx, rows, cols, tokens):
    rng = np.random.default_rng(rows + cols + tokens)
    words = orc.pack_f32((rng.standard_normal(rows * cols) * 0.02).astype(np.float32), rows, cols)[0]
    w = ctx.upload_ternary(words, rows, cols, 0.37)
    q = rng.integers(-128, 128, (tokens, cols)).astype(np.int8)
    amax = np.abs(rng.standard_normal(tokens)).astype(np.float32) + np.float32(0.1)
    bias, res = rng.standard_normal(rows).astype(np.float32), rng.standard_normal((tokens, rows)).astype(np.float32)
    dev = [ctx.to_device(a) for a in (q, amax, bias, res)]
    out, acc = ctx.alloc(tokens * rows * 4), ctx.alloc(tokens * rows * 4)
    ctx.ternary_linear(w, tokens, dev[0], dev[1], out, bias=dev[2], residual=dev[3], act=cabi.ACT_RELU2, acc_out=acc)
    sums = q.astype(np.float64) @ np_unpack(words, rows, cols).astype(np.float64).T
    assert (ctx.download(acc, (tokens, rows), np.int32) == sums.astype(np.int32)).all()
    f = (sums * (np.float64(np.float32(0.37)) * amax.astype(np.float64) / 127.0)[:, None] + bias.astype(np.float64)).astype(np.float32)
    f = np.where(f < 0, np.float32(0), f * f) + res
    assert (ctx.download(out, (tokens, rows), np.float32).view(np.uint32) == f.view(np.uint32)).all()
    for p in (*dev, out, acc):
        ctx.free(p)


@pytest.mark.parametrize("rows,cols", [(16, 128), (33, 1001), (2560, 6912), (300, 16500)])
@pytest.mark.parametrize("tokens", [3, 17, 30])
def test_dense_rows_are_quantized_alike(ctx, rows, cols, tokens):
    rng = np.random.default_rng(cols + tokens)
    m = orc.Matrix.from_f32((rng.standard_normal(rows * cols) * 0.02).astype(np.float32), rows, cols)
    w = ctx.upload_ternary(m.words, rows, cols, m.scale)
    x = rng.standard_normal((tokens, cols)).astype(np.float32)
    x[1] = 0
    pre, post = cabi.dense_forward(ctx, w, cabi.ACT_RELU, x)
    q, amax = orc.quantize_rows_f32(x)
    sums = q.astype(np.float64) @ np_unpack(m.words, rows, cols).astype(np.float64).T
    f = (sums * (np.float64(m.scale) * amax.astype(np.float64) / 127.0)[:, None]).astype(np.float32)
    assert (pre.view(np.uint32) == f.view(np.uint32)).all()
    assert (post == np.maximum(f, 0)).all()


@pytest.mark.parametrize("cols", [64, 1001, 16500])
def test_rows_that_are_not_numbers(ctx, cols):
    """Infinities, NaN, the largest and the smallest numbers in a pass of several tokens: the bits of a token by itself."""
    rng = np.random.default_rng(cols)
    rows = 70
    w = ctx.upload_ternary(*(lambda m: (m.words, rows, cols, m.scale))(orc.Matrix.from_f32((rng.standard_normal(rows * cols) * 0.02).astype(np.float32), rows, cols)))
    special = np.array([np.inf, -np.inf, np.nan, 3.4e38, -3.4e38, 1e-45, 0.0, -0.0, 1e-5, 9.9e-6], np.float32)
    x = rng.standard_normal((2 * len(special), cols)).astype(np.float32)
    for i, v in enumerate(special):
        x[2 * i, rng.integers(0, cols)] = v
        x[2 * i + 1] = v
    pre, post = cabi.dense_forward(ctx, w, cabi.ACT_LINEAR, x)
    for i in range(len(x)):
        one, _ = cabi.dense_forward(ctx, w, cabi.ACT_LINEAR, x[i:i + 1])
        assert (pre[i].view(np.uint32) == one[0].view(np.uint32)).all()


@pytest.mark.parametrize("heads,kvh,hd,inter,seq", [(4, 2, 32, 500, 23), (3, 1, 50, 130, 24), (20, 5, 128, 6912, 10), (2, 2, 2, 17, 29)])
def test_short_prompts_and_sequences_match_the_oracle(ctx, heads, kvh, hd, inter, seq):
    """A prompt in passes of 24 tokens, then 18 sequences of different lengths a token each per pass; logits as in test_gpu_batch.py."""
    rng = np.random.default_rng(inter)
    H, V, L, msl, B = heads * hd, 96, 2, 64, 18
    shapes = ((H, H), (kvh * hd, H), (kvh * hd, H), (H, H), (inter, H), (inter, H), (H, inter))
    dec = cabi.Decoder(ctx, L, H, heads, kvh, hd, inter, V, 1e-5, 10000.0, cabi.ACT_SILU, msl)
    many = cabi.Decoder(ctx, L, H, heads, kvh, hd, inter, V, 1e-5, 10000.0, cabi.ACT_SILU, msl) if H % 4 == 0 else None
    odec = orc.Decoder(L, H, heads, kvh, hd, inter, V, 1e-5, 10000.0, orc.ACT_SILU, msl)
    if many:
        many.set_batch(B)
    for b in range(L):
        packed = [orc.pack_f32((rng.standard_normal(r * c) * 0.02).astype(np.float32), r, c) for r, c in shapes]
        ws = [ctx.upload_ternary(p[0], r, c, p[1]) for p, (r, c) in zip(packed, shapes)]
        for d in filter(None, (dec, many)):
            d.set_block(b, ws)
        odec.set_block_packed(b, [p[0] for p in packed], [p[1] for p in packed])
    emb = (rng.standard_normal((V, H)) * 0.02).astype(np.float32)
    demb = ctx.to_device(emb)
    for d in filter(None, (dec, many)):
        d.set_embeddings(demb)
    odec.set_embeddings(emb)
    prompt = rng.integers(0, V, seq).astype(np.int32)
    want = odec.forward(prompt)
    tol = 1e-6 * max(1.0, float(np.max(np.abs(want))))
    assert np.max(np.abs(dec.forward(prompt) - want)) <= tol
    if many:
        starts = [rng.integers(0, V, 1 + i).astype(np.int32) for i in range(B)]
        for i, p in enumerate(starts):
            many.select(i)
            many.forward(p, want_logits=False)
        tok = rng.integers(0, V, B).astype(np.int32)
        got = many.step_batch(tok)
        for i, p in enumerate(starts):
            dec.reset()
            assert np.max(np.abs(got[i] - dec.forward(np.append(p, tok[i])))) <= tol
        many.close()
    dec.close()
