"""Logits on their way to the host: rows in pageable memory (large ones in pieces through pinned rows) are those that a caller's pinned
rows receive, for one row and for several passes of sequences, vocabularies of any size; one row is also held to the plain oracle.

Two decoders of the same weights take the same steps; whole rows are compared bit for bit.
"""
import numpy as np
import pytest
import torch

import donodra_oracle as do
import donodrakit as dk
import loom_b200
import stackkit as kit
from loom_b200 import cabi, models

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("vocab,batch", [(70, 2), (1023, 17), (120011, 9), (120011, 1), (300, 1)])
def test_pageable_and_pinned_rows_agree(vocab, batch):
    ctx = loom_b200.Context(0)
    cfg = dk.config(64, vocab, [dk.mlstm(2, 16, 24, 9.0, 48)])
    w = kit.Weights(dk.random_weights(cfg, 3))
    a, b = (models.build(ctx, cfg, w, models.LoadOptions(cabi.DTYPE_BF16, 16, batch)) for _ in range(2))
    pinned = torch.empty(batch, vocab, pin_memory=True)
    try:
        rng = np.random.default_rng(1)
        for i in range(batch):
            prompt = rng.integers(0, vocab, 3).astype(np.int32)
            for d in (a, b):
                d.select(i)
            assert np.array_equal(a.extend(prompt, [2])[0], b.extend(prompt, [0, 1, 2])[2])
        for _ in range(3):
            tok = rng.integers(0, vocab, batch).astype(np.int32)
            got = a.step_batch(tok) if batch > 1 else a.extend(tok, [0])
            if batch > 1:
                assert cabi.lib().loom_b200_decoder_step_batch(b.h, tok.ctypes.data, pinned.data_ptr()) == 0
            else:
                pinned.copy_(torch.from_numpy(b.extend(tok, [0])))
            assert np.array_equal(got, pinned.numpy())
    finally:
        a.close()
        b.close()
        ctx.close()


@pytest.mark.parametrize("vocab", [3, 70, 49151, 49152, 49153, 120011])  # (rows of 192 KB and more come in pieces)
@pytest.mark.parametrize("pinned", [False, True])
def test_one_row_against_the_oracle(vocab, pinned):
    """float32 weights: 2e-5 of the row as in test_gpu_donodra.py.  The row lies at an odd place in a larger buffer, whose other values stay."""
    ctx = loom_b200.Context(0)
    cfg = dk.config(40, vocab, [dk.mlstm(2, 16, 24, 9.0, 48)])
    w = dk.random_weights(cfg, 3)
    dec = models.build(ctx, cfg, kit.Weights(w), models.LoadOptions(cabi.DTYPE_F32, 16, 1))
    try:
        tok = np.random.default_rng(1).integers(0, vocab, 5).astype(np.int32)
        want, _ = do.forward(cfg, w, tok)
        buffer = torch.empty(vocab + 2000, pin_memory=pinned)
        at = 0
        for n, places in ((3, [2]), (1, [0]), (1, [0])):  # a prompt's last row, then single steps
            buffer.fill_(-7.0)
            here, place = np.ascontiguousarray(tok[at:at + n]), np.asarray(places, np.int32)
            ctx._check(cabi.lib().loom_b200_decoder_extend(dec.h, here.ctypes.data, n, place.ctypes.data, 1, buffer.data_ptr() + 4 * 777))
            got = buffer.numpy()
            assert kit.error(got[None, 777:777 + vocab], want[at + n - 1][None]).max() < 5 * 2e-5
            assert (got[:777] == -7).all() and (got[777 + vocab:] == -7).all()
            at += n
    finally:
        dec.close()
        ctx.close()
