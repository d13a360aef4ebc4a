"""The one-token products of a stack where their weight ring can go wrong: several strips of rows per CTA, fewer K slices than warps,
rows that leave room for one slot of the ring or for none, and the input rows' edges (columns beyond the registers of a thread,
rows that are no multiple of 16 bytes).

Every sequence of a batch is held to the plain oracle; tolerances as in test_gpu_donodra.py.
"""
import numpy as np
import pytest

import donodra_oracle as do
import donodrakit as dk
import loom_b200
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
