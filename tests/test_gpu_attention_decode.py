"""Attention of one new token per sequence over long KV rings: slices of a cluster that go through shared memory in chunks.

One decoder block over restored KV rings against the CPU oracle's.  Contexts end just before, at and after the places where a
slice (context / CTAs of the cluster) fills a chunk of 128 positions; ring lengths decide whether a slice can be longer than a
chunk at all.  Bound: all sums are float64 on both sides (relative error of a softmax sum of n terms below n * 2^-53 * cond,
1e-11 here), so rows differ by float32 rounding of the last step only: 1e-6 of the row maximum, as for the other layer tests.
"""
import numpy as np
import pytest

import loom_b200
from loom_b200 import cabi
from oracle import oracle as orc

pytestmark = pytest.mark.gpu
THREADS = min(16, orc.host_threads())


def run(heads, kvh, hd, msl, offsets, seed, **options):
    """One step of len(offsets) sequences, sequence i behind offsets[i] restored positions."""
    rng = np.random.default_rng(seed)
    ctx = loom_b200.Context(0)
    for name, value in options.items():
        ctx.set_option(name, value)
    H, inter, V, B = heads * hd, 256, 64, len(offsets)
    shapes = ((H, H), (kvh * hd, H), (kvh * hd, H), (H, H), (inter, H), (inter, H), (H, inter))
    packed = [orc.pack_f32((rng.standard_normal(r * c) * 0.02).astype(np.float32), r, c) for r, c in shapes]
    emb = (rng.standard_normal((V, H)) * 0.02).astype(np.float32)
    gdec = cabi.Decoder(ctx, 1, H, heads, kvh, hd, inter, V, 1e-5, 500000.0, cabi.ACT_SILU, msl)
    try:
        if B > 1:
            gdec.set_batch(B)
        gdec.set_block(0, [ctx.upload_ternary(p[0], r, c, p[1]) for p, (r, c) in zip(packed, shapes)])
        gdec.set_embeddings(ctx.to_device(emb))
        want, tokens = [], rng.integers(0, V, B).astype(np.int32)
        for i, n in enumerate(offsets):
            k = rng.standard_normal((n, kvh * hd)).astype(np.float32)
            v = rng.standard_normal((n, kvh * hd)).astype(np.float32)
            k[:, ::7] *= 3.0  # (peaked softmaxes: the running maximum moves from chunk to chunk)
            odec = orc.Decoder(1, H, heads, kvh, hd, inter, V, 1e-5, 500000.0, orc.ACT_SILU, msl)
            odec.set_block_packed(0, [p[0] for p in packed], [p[1] for p in packed])
            odec.set_embeddings(emb)
            odec.set_kv(0, n, k, v)
            want.append(odec.forward(tokens[i:i + 1], threads=THREADS))
            if B > 1:
                gdec.select(i)
            gdec.upload_cache(0, n, k, v)
        got = gdec.step_batch(tokens) if B > 1 else gdec.forward(tokens)[None]
        for g, w in zip(got, want):
            assert np.max(np.abs(g - w)) <= 1e-6 * max(1.0, float(np.max(np.abs(w))))
    finally:
        gdec.close()
        ctx.close()


@pytest.mark.parametrize("heads,kvh,hd", [(2, 2, 128), (4, 2, 128), (4, 1, 128), (8, 1, 128), (8, 2, 48), (16, 2, 64)])
@pytest.mark.parametrize("msl,context", [(9000, 1), (9000, 2046), (9000, 2047), (9000, 2048), (9000, 4111), (3000, 2999)])
def test_one_sequence(heads, kvh, hd, msl, context):
    run(heads, kvh, hd, msl, [context], context)


@pytest.mark.parametrize("heads,kvh,hd,msl,offsets", [
    (4, 1, 128, 9000, [2046, 1, 5000]),                       # clusters of sixteen
    (8, 8, 128, 3000, [1, 254, 255, 256, 300, 2, 700, 511]),  # pairs of CTAs
    (32, 8, 64, 6000, [126, 127, 128, 1, 2500, 3, 4, 5]),
    (8, 1, 128, 9000, [4095] * 2),
    (64, 8, 80, 5000, [1, 2047, 300, 4000, 5, 130, 64, 2]),  # eight heads as two times four, 16 pairs of clusters
    (16, 2, 80, 12000, [3000, 1, 9001]),
    (16, 16, 64, 4000, [127, 128, 129, 1, 400, 2, 3, 256, 5, 600, 1]),  # single CTAs, then a pass of three
])
def test_several_sequences(heads, kvh, hd, msl, offsets):
    run(heads, kvh, hd, msl, offsets, len(offsets))


@pytest.mark.parametrize("options", [dict(attn_cluster=0), dict(fold_rope=0), dict(attn_cluster=0, decode_splits=1)], ids=["cluster off", "rotation apart", "one split"])
@pytest.mark.parametrize("heads,kvh,hd,msl", [(4, 1, 128, 61000), (8, 1, 128, 130000), (16, 16, 64, 105000)])
def test_several_sequences_without_the_cluster_kernel(options, heads, kvh, hd, msl):
    """Rings of which a quarter is more than a CTA's scores have room for (59,900 positions at head dimension 128)."""
    run(heads, kvh, hd, msl, [20000, 1, 640], heads, **options)
