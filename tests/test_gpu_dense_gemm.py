"""The token-block products of a stack over few tiles (with plain multiply-adds the CTAs of a cluster share a tile's K slices), ragged rows,
columns and tokens, and every epilogue (gate, gelu, residual, image, per-head blocks).

Logits of a whole prompt against the plain oracles; tolerances as in test_gpu_donodra.py and test_gpu_stack.py.
"""
import numpy as np
import pytest

import donodra_oracle as do
import donodrakit as dk
import loom_b200
import stack_oracle as so
import stackkit as kit
from loom_b200 import cabi, models

pytestmark = pytest.mark.gpu
F32, BF16 = cabi.DTYPE_F32, cabi.DTYPE_BF16


@pytest.fixture(scope="module")
def ctx():
    c = loom_b200.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("dtype,tensor_cores", [(F32, 1), (BF16, 1), (BF16, 0)], ids=["f32", "bf16", "bf16-plain"])
@pytest.mark.parametrize("width,ff,tokens", [(700, 1500, 130), (1100, 2610, 33), (520, 1030, 300), (264, 4100, 9)])
def test_prompts_over_few_tiles(ctx, dtype, tensor_cores, width, ff, tokens):
    ctx.set_option("dense_tc", tensor_cores)
    try:
        for cfg, weights, oracle, tol in (
                (dk.config(width, 150, [dk.mlstm(2, 40, 136, 9.0, ff), dk.attention(4, 2, 48, 40, 512, 90.0, 0.15, None)]), dk.random_weights, do.forward, 0.02),
                (kit.config(width, 150, [kit.latent(3, 48, 56, 72, 0.14, kit.dense(ff)), kit.gla(2, 40, 136, 8.0, None)]), kit.random_weights, so.forward, 0.06)):
            w = weights(cfg, 7)
            dec = models.build(ctx, cfg, kit.Weights(w), models.LoadOptions(dtype, 512, 1))
            tok = np.random.default_rng(tokens).integers(0, 150, tokens).astype(np.int32)
            want, _ = oracle(cfg, w, tok)
            first = dec.extend(tok, range(tokens))
            e = kit.error(first, want)
            tol = 2e-5 if dtype == F32 else tol
            assert np.quantile(e, 0.9) < tol and e.max() < 5 * tol
            dec.reset()
            assert np.array_equal(dec.extend(tok, range(tokens)), first)  # the parts of a tile meet in the order of K
            dec.close()
    finally:
        ctx.set_option("dense_tc", 1)


@pytest.mark.parametrize("width,ff,tokens", [(1300, 2100, 1500), (2560, 700, 600), (640, 5000, 2100), (330, 1000, 1030)])
def test_tiles_of_any_width(ctx, width, ff, tokens):
    """Prompts of many tiles, whose columns are cut where the waves of CTAs come out even: across blocks of 128 rows of a matrix, with
    ragged last ones; whole models against the plain multiply-adds, with the tolerances to the oracle above (each side is within them).
    A wrong group of columns may hide in such a row's error: test_gpu_gemm_bf16.py has the products column by column."""
    for cfg, weights, tol in (
            (dk.config(width, 96, [dk.mlstm(2, 40, 136, 9.0, ff), dk.attention(4, 2, 48, 40, 512, 90.0, 0.15, ff)]), dk.random_weights, 0.02),
            (kit.config(width, 96, [kit.latent(3, 48, 56, 72, 0.14, kit.dense(ff)), kit.gla(2, 40, 136, 8.0, kit.dense(ff))]), kit.random_weights, 0.06)):
        dec = models.build(ctx, cfg, kit.Weights(weights(cfg, 11)), models.LoadOptions(BF16, tokens, 1))
        tok = np.random.default_rng(tokens).integers(0, 96, tokens).astype(np.int32)
        places = range(0, tokens, 37)
        got = []
        for tensor_cores in (1, 0):
            ctx.set_option("dense_tc", tensor_cores)
            try:
                dec.reset()
                got.append(dec.extend(tok, places))
            finally:
                ctx.set_option("dense_tc", 1)
        e = kit.error(got[0], got[1])
        assert np.quantile(e, 0.9) < 2 * tol and e.max() < 10 * tol
        dec.close()
