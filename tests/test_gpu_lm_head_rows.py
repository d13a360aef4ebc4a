"""The fp32 head for several sequences in one pass over the table (float64 matrix instructions): every sequence's logits and greedy
token against the CPU oracle, at the edges of its tiles: fewer vocabulary rows than a strip of 32 or than CTAs, shares that end
inside a strip, hidden sizes that are no multiple of the 16-column step, two to eight rows, the largest hidden size.

Bound: products of float32 values are exact in float64 and K <= 5504 of them add up with a relative error below K * 2^-53 =
7e-13 of the sum of magnitudes, far below half a float32 unit: logits agree to 1e-6 of the largest.
"""
import numpy as np
import pytest

import loom_b200
from loom_b200 import cabi
from oracle import oracle as orc

pytestmark = pytest.mark.gpu
THREADS = min(16, orc.host_threads())


@pytest.mark.parametrize("heads,hd,V,B", [(2, 64, 20, 2), (2, 64, 5003, 8), (4, 65 * 4, 4736 + 33, 7), (1, 84, 300, 3), (9, 100, 32 * 148 + 1, 5), (2, 50 * 4, 1025, 11),
                                          (43, 128, 700, 8), (40, 128, 128, 6)])
def test_rows_per_pass(heads, hd, V, B):
    rng = np.random.default_rng(V + B)
    ctx = loom_b200.Context(0)
    H, inter, msl = heads * hd, 128, 16
    shapes = ((H, H), (hd, H), (hd, H), (H, H), (inter, H), (inter, H), (H, inter))
    packed = [orc.pack_f32((rng.standard_normal(r * c) * 0.02).astype(np.float32), r, c) for r, c in shapes]
    emb = (rng.standard_normal((V, H)) * 0.02).astype(np.float32)
    emb[V // 2] = emb[V // 3]  # equal rows give equal logits: the first maximum counts
    gain = (1 + 0.1 * rng.standard_normal(H)).astype(np.float32)
    gdec = cabi.Decoder(ctx, 1, H, heads, 1, hd, inter, V, 1e-5, 500000.0, cabi.ACT_SILU, msl)
    try:
        gdec.set_batch(B)
        gdec.set_block(0, [ctx.upload_ternary(p[0], r, c, p[1]) for p, (r, c) in zip(packed, shapes)])
        gdec.set_embeddings(ctx.to_device(emb), gain)
        odecs = []
        for i in range(B):
            od = orc.Decoder(1, H, heads, 1, hd, inter, V, 1e-5, 500000.0, orc.ACT_SILU, msl)
            od.set_block_packed(0, [p[0] for p in packed], [p[1] for p in packed])
            od.set_embeddings(emb, gain)
            prompt = rng.integers(0, V, 1 + i % 3).astype(np.int32)
            od.forward(prompt, threads=THREADS)
            odecs.append(od)
            gdec.select(i)
            gdec.forward(prompt)
        tokens = rng.integers(0, V, B).astype(np.int32)
        got = gdec.step_batch(tokens)
        want = [od.forward(tokens[i:i + 1], threads=THREADS) for i, od in enumerate(odecs)]
        for g, w in zip(got, want):
            assert np.max(np.abs(g - w)) <= 1e-6 * max(1.0, float(np.max(np.abs(w))))
        gdec.continue_batch(2)
        first = gdec.generated_tokens_batch(2)[:, 0]
        assert first.tolist() == [int(orc.argmax(g)) for g in got]
    finally:
        gdec.close()
        ctx.close()
