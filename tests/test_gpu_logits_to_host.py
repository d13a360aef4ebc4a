"""Logits on their way to the host: rows in pageable memory (pieces through pinned rows, shared out to threads when they are large) are
those that a caller's pinned rows receive, for one row and for several passes of sequences, vocabularies of any size.

Two decoders of the same weights take the same steps; whole rows are compared bit for bit.
"""
import numpy as np
import pytest
import torch

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
