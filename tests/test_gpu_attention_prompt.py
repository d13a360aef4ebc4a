"""Float64 attention and rotation of a prompt block: query heads per KV head from one to 64,
head dimensions, and prompts that end just before, at and after a tile of keys or of query rows.

Two decoder blocks against the CPU oracle's: the second block's keys carry every row of the first one's attention.  All sums are
float64 on both sides, so logits differ by float32 rounding of the last step only: 1e-6 of the row maximum, as in
test_gpu_attention_decode.py.
"""
import numpy as np
import pytest

import loom_b200
from loom_b200 import cabi
from oracle import oracle as orc

pytestmark = pytest.mark.gpu
THREADS = min(16, orc.host_threads())


@pytest.mark.parametrize("heads,kvh,hd,prompts", [(4, 4, 128, (32, 33)), (4, 2, 64, (63, 64)), (8, 2, 48, (65, 96)), (8, 1, 16, (97, 31 + 8)), (16, 1, 32, (40,)),
                                                  (32, 1, 16, (35, 64)), (64, 1, 16, (33, 70)), (4, 1, 128, (129, 7, 32)),
                                                  (24, 8, 16, (129, 127)), (40, 10, 16, (85,)), (12, 4, 32, (256,))])
def test_prompts_match_the_oracle(heads, kvh, hd, prompts):
    rng = np.random.default_rng(heads + hd)
    ctx = loom_b200.Context(0)
    H, inter, V, L, msl = heads * hd, 320, 64, 2, 256
    shapes = ((H, H), (kvh * hd, H), (kvh * hd, H), (H, H), (inter, H), (inter, H), (H, inter))
    emb = (rng.standard_normal((V, H)) * 0.02).astype(np.float32)
    gdec = cabi.Decoder(ctx, L, H, heads, kvh, hd, inter, V, 1e-5, 500000.0, cabi.ACT_SILU, msl)
    odec = orc.Decoder(L, H, heads, kvh, hd, inter, V, 1e-5, 500000.0, orc.ACT_SILU, msl)
    try:
        for b in range(L):
            packed = [orc.pack_f32((rng.standard_normal(r * c) * 0.02).astype(np.float32), r, c) for r, c in shapes]
            gdec.set_block(b, [ctx.upload_ternary(p[0], r, c, p[1]) for p, (r, c) in zip(packed, shapes)])
            odec.set_block_packed(b, [p[0] for p in packed], [p[1] for p in packed])
        gdec.set_embeddings(ctx.to_device(emb))
        odec.set_embeddings(emb)
        for n in prompts:  # one after the other, over the rows of the one before
            tok = rng.integers(0, V, n).astype(np.int32)
            got, want = gdec.forward(tok), odec.forward(tok, threads=THREADS)
            assert np.max(np.abs(got - want)) <= 1e-6 * max(1.0, float(np.max(np.abs(want))))
    finally:
        gdec.close()
        ctx.close()


@pytest.mark.parametrize("heads,kvh,hd,n", [(24, 8, 64, 128), (24, 8, 64, 137), (7, 1, 48, 512), (20, 5, 128, 165), (20, 5, 16, 500), (64, 8, 80, 57), (35, 7, 128, 99)])
def test_rotation_of_a_block_in_any_share(heads, kvh, hd, n):
    """From 4096 (token, head) pairs on a token's angles are computed once and its heads shared out; two halves of the prompt lie below
    that.  The first block's keys are rotated projections of the tokens alone: the same bits either way."""
    rng = np.random.default_rng(n)
    ctx = loom_b200.Context(0)
    H, inter, V, msl = heads * hd, 128, 64, 640
    shapes = ((H, H), (kvh * hd, H), (kvh * hd, H), (H, H), (inter, H), (inter, H), (H, inter))
    dec = cabi.Decoder(ctx, 1, H, heads, kvh, hd, inter, V, 1e-5, 500000.0, cabi.ACT_SILU, msl)
    try:
        packed = [orc.pack_f32((rng.standard_normal(r * c) * 0.02).astype(np.float32), r, c) for r, c in shapes]
        dec.set_block(0, [ctx.upload_ternary(p[0], r, c, p[1]) for p, (r, c) in zip(packed, shapes)])
        dec.set_embeddings(ctx.to_device((rng.standard_normal((V, H)) * 0.02).astype(np.float32)))
        tok = rng.integers(0, V, n).astype(np.int32)
        rows = []
        for parts in ((tok,), (tok[:n // 2], tok[n // 2:])):
            dec.reset()
            logits = [dec.extend(t, [len(t) - 1])[0] for t in parts][-1]
            k, v = np.zeros((msl, kvh * hd), np.float32), np.zeros((msl, kvh * hd), np.float32)
            ctx._check(cabi.lib().loom_b200_decoder_download_cache(dec.h, 0, k.ctypes.data, v.ctypes.data))
            rows.append((k[:n], logits))
        (k0, l0), (k1, l1) = rows
        assert k0.any(axis=1).all() and np.array_equal(k0, k1)
        assert np.max(np.abs(l0 - l1)) <= 1e-6 * max(1.0, float(np.max(np.abs(l1))))
    finally:
        dec.close()
        ctx.close()
