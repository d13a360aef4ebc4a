"""Float64 attention and rotation of a prompt block: query heads per KV head from one to 64,
head dimensions, and prompts that end just before, at and after a tile of keys or of query rows.

Two decoder blocks against the CPU oracle's: the second block's keys carry every row of the first one's attention.  All sums are
float64 on both sides, so logits differ by float32 rounding of the last step only: 1e-6 of the row maximum, as in
test_gpu_attention_decode.py.
"""
import numpy as np
import pytest

import harness
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


@pytest.mark.parametrize("heads,kvh,hd,tokens,pos0", [(8, 2, 128, 150, 0), (4, 4, 64, 97, 40), (20, 5, 128, 33, 130)])
def test_infinities_and_nan_stay_with_the_rows_that_see_them(heads, kvh, hd, tokens, pos0):
    """Keys and values that are not finite, in float64 as IEEE has them: a NaN score makes a NaN row, so does one of +infinity, one of -infinity
    weighs nothing.  A position's value also reaches rows in front of it in its tile of 32 keys, with weight zero; those are left out where
    the value is not finite."""
    rng = np.random.default_rng(tokens)
    msl, G = 320, heads // kvh
    ctx = loom_b200.Context(0)
    try:
        for special in ("none", "key nan", "key inf", "key -inf", "value inf", "value nan", "query nan", "lowest"):
            q = rng.standard_normal((tokens, heads, hd))
            k, v = (rng.standard_normal((kvh, msl, hd)).astype(np.float32) for _ in range(2))
            at = pos0 + tokens // 2
            what = special.split()
            if what[0] in ("key", "value"):
                (k if what[0] == "key" else v)[0, at, 3] = np.float32(what[1])
            if special.startswith("key"):
                q[..., 3] = np.abs(q[..., 3]) + 0.1  # (infinite scores of one sign)
            if special == "query nan":
                q[tokens // 3, 1, 5] = np.nan
            if special == "lowest":
                k[:, at:at + 2] = np.finfo(np.float32).min
            if pos0 + tokens < msl:  # what lies behind the block is nobody's
                k[:, pos0 + tokens:], v[:, pos0 + tokens:] = np.nan, np.inf
            dev = [ctx.to_device(a) for a in (q, k, v, np.array([pos0], np.int32))]
            dout = ctx.alloc(tokens * heads * hd * 8)
            ctx._check(harness.lib().t_attention_prompt(ctx.h, *dev, dout, tokens, heads, kvh, hd, msl))
            got = ctx.download(dout, (tokens, heads, hd), np.float64)
            for h in range(heads):
                kk, vv = k[h // G].astype(np.float64), v[h // G].astype(np.float64)
                for t in range(tokens):
                    pos = pos0 + t
                    if what[0] == "value" and h < G and at // 32 * 32 <= pos < at:
                        continue
                    with np.errstate(all="ignore"):
                        s = (kk[:pos + 1] * q[t, h]).sum(1) / np.sqrt(hd)
                        e = np.exp(s - s.max()) if not np.isnan(s).any() else np.full(pos + 1, np.nan)
                        want = (e[:, None] * vv[:pos + 1]).sum(0) / e.sum()
                    bad = ~np.isfinite(want)
                    assert np.array_equal(np.isnan(got[t, h]), np.isnan(want)) and np.array_equal(got[t, h][bad & ~np.isnan(want)], want[bad & ~np.isnan(want)])
                    # a score of up to 40 is off by 128 * 40 * 2^-53 = 6e-13 at most, and its weight by as much of itself
                    if not bad.all():
                        terms = (e[:, None] * np.abs(vv[:pos + 1])).sum(0) / e.sum()
                        assert (np.abs(got[t, h][~bad] - want[~bad]) <= 1e-12 * terms[~bad]).all()
            for p in (*dev, dout):
                ctx.free(p)
    finally:
        ctx.close()
