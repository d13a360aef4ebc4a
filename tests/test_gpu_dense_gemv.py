"""The one-token products of a stack where their weight ring can go wrong: several strips of rows per CTA, fewer K slices than warps,
rows that leave room for one slot of the ring or for none, and the input rows' edges (columns beyond the registers of a thread, for
every prologue, rows that are no multiple of 16 bytes).

Every sequence of a batch is held to the plain oracle; tolerances as in test_gpu_donodra.py and test_gpu_stack.py.
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
TOL = {F32: 2e-5, BF16: 0.02}


@pytest.fixture(scope="module")
def ctx():
    c = loom_b200.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("dtype,width,ff,vocab,batch", [
    (BF16, 64, 5000, 9500, 1), (F32, 32, 2500, 9500, 2), (BF16, 200, 4800, 70, 3), (F32, 77, 4801, 70, 1),
    (BF16, 25536, 24, 70, 4),  # 204,288 B of input rows: one slot of the single ring, none of the double one
    (BF16, 64, 12500, 70, 8), (F32, 32, 12400, 70, 4), (BF16, 40, 24600, 70, 3),  # the same for the second product's rows
    (BF16, 17000, 40, 70, 1), (F32, 12768, 24, 70, 4), (F32, 8500, 40, 70, 1)])
def test_steps_of_wide_and_narrow_stacks(ctx, dtype, width, ff, vocab, batch):
    cfg = dk.config(width, vocab, [dk.mlstm(2, 8, 24, 9.0, ff), dk.attention(2, 1, 16, 16, 32, 9.0, 0.3, None)])
    w = dk.random_weights(cfg, 5)
    dec = models.build(ctx, cfg, kit.Weights(w), models.LoadOptions(dtype, 16, batch))
    tok = np.random.default_rng(2).integers(0, vocab, (batch, 5)).astype(np.int32)
    for i in range(batch):
        dec.select(i)
        dec.extend(tok[i, :2])
    got = []
    for j in range(2, 5):
        got.append(np.array(dec.step_batch(tok[:, j]) if batch > 1 else dec.extend(tok[:, j], [0])))
    for i in range(batch):
        want, _ = do.forward(cfg, w, tok[i])
        assert kit.error(np.stack([g[i] for g in got]), want[2:]).max() < 5 * TOL[dtype], i
    dec.close()


def normalised(row, gain, eps, threads):
    """A row through the norm of the prologue, operation by operation: thread i of `threads` adds the squares of columns i, i + threads, ...
    in that order, then a warp's 32 sums meet pairwise from afar to near, then the warps' in order.  (The product and sum of a fused
    multiply-add are exact in 64 bits of mantissa up to one rounding of the sum's last bits.)"""
    x = np.zeros(-(-len(row) // threads) * threads, np.float32)
    x[:len(row)] = row
    ss = np.zeros(threads, np.float32)
    for part in x.reshape(-1, threads):
        ss = (part.astype(np.longdouble) ** 2 + ss).astype(np.float32)
    ss = ss.reshape(-1, 32)
    for o in (16, 8, 4, 2, 1):
        ss = ss + ss[:, np.arange(32) ^ o]
    total = np.float32(0)
    for v in ss[:, 0]:
        total = total + v
    rstd = np.float32(1) / np.sqrt(total / np.float32(len(row)) + np.float32(eps))
    return row * rstd * np.float32(1) * gain


@pytest.mark.parametrize("width,batch", [(2560, 1), (2560, 2), (2560, 3), (1111, 1), (1111, 2), (40, 5), (6200, 1), (6200, 2)])
def test_norm_adds_columns_in_one_order(ctx, width, batch):
    """The last bits of a norm decide which way bf16 rounds a row, and that travels through the layers that follow: the sum's order is
    part of the result.  The embeddings' first rows are those of the unit matrix, so that the tied head hands out the normalised row."""
    def edit(w):
        w["embed"][:width] = np.eye(width)

    cfg = dk.config(width, width + 16, [dk.mlstm(2, 8, 24, 9.0, None)])
    w = dk.random_weights(cfg, 8, edit=edit)
    dec = models.build(ctx, cfg, kit.Weights(w), models.LoadOptions(F32, 16, batch))
    tok = np.random.default_rng(3).integers(width, width + 16, batch).astype(np.int32)
    for i in range(batch):
        dec.select(i)
        dec.extend(tok[i:i + 1])
    got = dec.step_batch(tok) if batch > 1 else dec.extend(tok, [0])
    rows = dec.last_residual(batch)
    for g, row in zip(np.asarray(got), rows):
        want = normalised(row[:width], np.asarray(w["final.norm"], np.float32), cfg["norm"]["eps"], 128 if batch == 2 else 256)
        assert np.array_equal(g[:width], want)
    dec.close()


@pytest.mark.parametrize("dtype,batch,ff", [(F32, 1, 40), (F32, 5, 40), (F32, 8, 200), (BF16, 1, 40)])
def test_infinite_weights_of_an_expert_stay_with_its_tokens(ctx, dtype, batch, ff):
    """One routed layer whose expert e has infinite weights in its second product: exactly the tokens that chose e lose their logits, and
    those of the others keep every bit.  (In bf16 matrix instructions multiply the tokens of a pass that did not choose with zeros.)"""
    E, top = 5, 2
    cfg = kit.config(72, 90, [kit.gla(2, 16, 24, 8.0, kit.moe(ff, E, top))])
    w = kit.random_weights(cfg, 4)
    tok = np.random.default_rng(6).integers(0, 90, (2, batch)).astype(np.int32)

    def logits(weights):
        dec = models.build(ctx, cfg, kit.Weights(weights), models.LoadOptions(dtype, 16, batch))
        for i in range(batch):
            dec.select(i)
            dec.extend(tok[0, i:i + 1])
        got = np.array(dec.step_batch(tok[1]) if batch > 1 else dec.extend(tok[1], [0]))
        dec.close()
        return got

    clean, chosen = logits(w), np.zeros(batch, int)
    for e in range(E):
        name = "l0.mlp.e%d.down" % e
        got = logits({**w, name: np.full_like(w[name], np.inf)})
        lost = ~np.isfinite(got).all(axis=1)
        assert np.array_equal(got[~lost], clean[~lost])
        chosen += lost
    assert np.array_equal(chosen, np.full(batch, top))


@pytest.mark.parametrize("dtype,width,heads,vdim,taps,batch", [
    (F32, 2100, 17, 128, 4, 1), (F32, 1100, 9, 128, 3, 2), (F32, 2100, 11, 200, 2, 3),  # registers hold 2048 columns of a row, 1024 with two
    (F32, 1101, 3, 700, 5, 2), (BF16, 4200, 17, 256, 4, 1), (BF16, 2120, 17, 128, 7, 2), (BF16, 4200, 9, 472, 4, 3)])  # 4096 and 2048
def test_convolved_and_gated_rows_beyond_the_registers(ctx, dtype, width, heads, vdim, taps, batch):
    """A convolution over the input rows and head norms with gates in front of the output product, both longer than what a thread keeps."""
    cfg = kit.config(width, 70, [kit.gla(heads, 16, vdim, 8.0, kit.dense(40)), kit.gla(1, 16, 24, 8.0, None)], taps=taps)
    w = kit.random_weights(cfg, 9)
    dec = models.build(ctx, cfg, kit.Weights(w), models.LoadOptions(dtype, 16, batch))
    tok = np.random.default_rng(4).integers(0, 70, (batch, 8)).astype(np.int32)
    for i in range(batch):
        dec.select(i)
        dec.extend(tok[i, :1])
    got = [np.array(dec.step_batch(tok[:, j]) if batch > 1 else dec.extend(tok[:, j], [0])) for j in range(1, 8)]
    for i in range(batch):
        want, _ = so.forward(cfg, w, tok[i])
        e = kit.error(np.stack([g[i] for g in got]), want[1:])
        assert np.quantile(e, 0.9) < {F32: 2e-5, BF16: 0.06}[dtype] and e.max() < 5 * {F32: 2e-5, BF16: 0.06}[dtype], i
    dec.close()
