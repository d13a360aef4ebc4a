"""Decode attention of several sequences whose rings are too long for a slice to be held at once: scores of a whole slice, softmax, values,
through a ring of four tiles of 64 positions.  Contexts that end before, at and behind a tile and behind the ring of tiles, slices that are
empty, eight heads per KV head as two groups of four; and rings too long for a slice's scores, which take the chunks.  Every sequence
against an oracle decoder of its own; all sums are float64 on both sides, so logits differ by float32 rounding of the last step only."""
import numpy as np
import pytest

import loom_b200
from loom_b200 import cabi
from oracle import oracle as orc

pytestmark = pytest.mark.gpu
THREADS = min(16, orc.host_threads())


@pytest.mark.parametrize("heads,kvh,hd,msl,most,prompts", [(8, 2, 128, 600, 2, (1, 63, 64, 126, 127)), (8, 2, 128, 1024, 2, (2, 65, 510, 513, 700)),
                                                           (8, 1, 64, 1200, 2, (3, 129, 600)), (4, 1, 128, 4000, 2, (5, 257, 400)), (4, 1, 128, 7000, 2, (5, 300)),
                                                           (4, 1, 112, 4096, 16, (1, 15, 16, 17, 1030))])
def test_sequences_over_long_rings(heads, kvh, hd, msl, most, prompts):
    rng = np.random.default_rng(heads + msl)
    ctx = loom_b200.Context(0)
    ctx.set_option("attn_cluster", most)
    H, inter, V, L = heads * hd, 192, 64, 2
    shapes = ((H, H), (kvh * hd, H), (kvh * hd, H), (H, H), (inter, H), (inter, H), (H, inter))
    emb = (rng.standard_normal((V, H)) * 0.02).astype(np.float32)
    gdec = cabi.Decoder(ctx, L, H, heads, kvh, hd, inter, V, 1e-5, 500000.0, cabi.ACT_SILU, msl)
    odecs = [orc.Decoder(L, H, heads, kvh, hd, inter, V, 1e-5, 500000.0, orc.ACT_SILU, msl) for _ in prompts]
    try:
        gdec.set_batch(len(prompts))
        for b in range(L):
            packed = [orc.pack_f32((rng.standard_normal(r * c) * 0.02).astype(np.float32), r, c) for r, c in shapes]
            gdec.set_block(b, [ctx.upload_ternary(p[0], r, c, p[1]) for p, (r, c) in zip(packed, shapes)])
            for od in odecs:
                od.set_block_packed(b, [p[0] for p in packed], [p[1] for p in packed])
        gdec.set_embeddings(ctx.to_device(emb))
        for i, (n, od) in enumerate(zip(prompts, odecs)):
            od.set_embeddings(emb)
            tok = rng.integers(0, V, n).astype(np.int32)
            od.forward(tok, threads=THREADS)
            gdec.select(i)
            gdec.forward(tok)
        for _ in range(4):
            tok = rng.integers(0, V, len(prompts)).astype(np.int32)
            got = gdec.step_batch(tok)
            for i, od in enumerate(odecs):
                want = od.forward(tok[i:i + 1], threads=THREADS)
                assert np.max(np.abs(got[i] - want)) <= 1e-6 * max(1.0, float(np.max(np.abs(want))))
    finally:
        gdec.close()
        ctx.close()
