"""Recorded frames beside calls that need more scratch than the frame does: what a frame uses stays allocated, so a replay computes the
same bits and writes nothing that belongs to somebody else by then."""
import numpy as np
import pytest

import loom_b200
from loom_b200 import cabi
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def matrix(ctx, rng, rows, cols):
    words, scale = orc.pack_f32((rng.standard_normal(rows * cols) * 0.02).astype(np.float32), rows, cols)
    return ctx.upload_ternary(words, rows, cols, scale)


@pytest.mark.parametrize("kind,tokens", [("linear", 1), ("linear", 4), ("linear", 20), ("gemm", 40)])
def test_replay_behind_a_wider_call(kind, tokens):
    rng = np.random.default_rng(tokens)
    ctx = loom_b200.Context(0)
    ctx.set_option("gemv_partition", 1 if tokens == 1 else 0)  # (one token: partial sums through the scratch)
    try:
        def call(rows, cols, n):
            w, x = matrix(ctx, rng, rows, cols), ctx.to_device(rng.standard_normal((n, cols)).astype(np.float32))
            q, amax, out = ctx.alloc(n * cols), ctx.alloc(n * 4), ctx.alloc(n * rows * 4)

            def run():
                if kind == "gemm":
                    ctx.ternary_gemm(w, n, x, out=out)
                else:
                    ctx.quantize_activation(n, cols, x, q, amax)
                    ctx.ternary_linear(w, n, q, amax, out)
            return run, out, w, (n, rows)

        run, out, _w, shape = call(300, 1000, tokens)
        run()
        ctx.sync()
        ctx.graph_begin()
        run()
        frame = ctx.graph_end()
        ctx.graph_launch(frame)
        want = ctx.download(out, shape, np.float32)
        wide, _, _w2, _ = call(20000, 4000, 24 if kind == "linear" else 600)
        wide()
        ctx.sync()
        # memory that a freed scratch would be part of by now
        mark = np.full(1 << 16, 0xA5, np.uint8)
        marks = [ctx.to_device(mark) for _ in range(200)]
        ctx.zero(out, int(np.prod(shape)) * 4)
        for _ in range(3):
            ctx.graph_launch(frame)
        assert np.array_equal(ctx.download(out, shape, np.float32).view(np.uint32), want.view(np.uint32))
        assert all((ctx.download(m, mark.shape, np.uint8) == mark).all() for m in marks)
        ctx.graph_free(frame)
        run()
        assert np.array_equal(ctx.download(out, shape, np.float32).view(np.uint32), want.view(np.uint32))
    finally:
        ctx.close()


@pytest.mark.parametrize("more", [2, 5, 24, 31])
def test_generation_behind_a_short_prompt(more):
    """A prompt, greedy tokens (their step is recorded, with a feed-forward wide enough to be quantized through the scratch), some more tokens
    in passes that need more of it, greedy tokens again."""
    rng = np.random.default_rng(more)
    L, H, heads, kvh, hd, inter, V, msl = 2, 128, 4, 2, 32, 8208, 96, 128
    ctx = loom_b200.Context(0)
    gdec = cabi.Decoder(ctx, L, H, heads, kvh, hd, inter, V, 1e-5, 10000.0, cabi.ACT_SILU, msl)
    odec = orc.Decoder(L, H, heads, kvh, hd, inter, V, 1e-5, 10000.0, orc.ACT_SILU, msl)
    try:
        for b in range(L):
            shapes = ((H, H), (kvh * hd, H), (kvh * hd, H), (H, H), (inter, H), (inter, H), (H, inter))
            packed = [orc.pack_f32((rng.standard_normal(r * c) * 0.02).astype(np.float32), r, c) for r, c in shapes]
            gdec.set_block(b, [ctx.upload_ternary(p[0], r, c, p[1]) for p, (r, c) in zip(packed, shapes)])
            odec.set_block_packed(b, [p[0] for p in packed], [p[1] for p in packed])
        emb = (rng.standard_normal((V, H)) * 0.02).astype(np.float32)
        gdec.set_embeddings(ctx.to_device(emb))
        odec.set_embeddings(emb)
        for tokens, steps in ((40, 3), (more, 3)):
            tok = rng.integers(0, V, tokens).astype(np.int32)
            want, got = odec.forward(tok), gdec.forward(tok)
            for s in range(steps + 1):
                assert np.max(np.abs(got - want)) <= 1e-6 * max(1.0, float(np.max(np.abs(want))))
                if s < steps:
                    nxt = np.array([int(np.argmax(want))], np.int32)
                    want, got = odec.forward(nxt), gdec.forward(nxt)
    finally:
        gdec.close()
        ctx.close()
