"""Norm with convolution of a block of tokens: one, two or four tokens to a CTA by the block's length.  Lengths that leave a rest in the last
CTA, rows with and without 16-byte loads, from one tap to more taps than a CTA has tokens, behind an empty ring and behind the tokens of a
portion before; against the oracle, to the bounds of the stacks' other tests."""
import numpy as np
import pytest

import stackkit as kit
import test_gpu_stack as ts
from test_gpu_stack import ctx  # noqa: F401 (fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,taps", [(56, 4), (77, 7), (64, 1), (40, 2)])
@pytest.mark.parametrize("dtype", [ts.F32, ts.BF16], ids=["f32", "bf16"])
def test_tokens_of_a_cta(ctx, width, taps, dtype):  # noqa: F811
    cfg = kit.config(width, 70, [kit.gla(1, 8, 8, 4.0, None)], taps=taps)
    m = ts.Model(ctx, cfg, 21, dtype, max_seq=640)
    try:
        tok = ts.tokens_of(cfg, 600, 3)
        want, _ = m.oracle(tok)
        for n in (297, 593, 595):  # two tokens a CTA from 296 tokens on, four from 592
            assert ts.close(cfg, dtype, m.whole(tok[:n]), want[:n])
        assert ts.close(cfg, dtype, m.cut(tok, [3, 595, 2]), want)
        assert ts.close(cfg, dtype, m.cut(tok, [300]), want)
    finally:
        m.close()
