"""Host rows of the layer calls.  They cross in slots of 128 KB, eight in flight: the sizes are a slot's edges and more than the eight, in
and out.  Pinned memory of the caller is copied as it is.  The sums are whole numbers with one rescale: the oracle's bits."""
import threading

import numpy as np
import pytest
import torch

import loom_b200
from loom_b200 import cabi
from oracle import oracle as orc

pytestmark = pytest.mark.gpu
SLOT = 128 * 1024 // 4  # floats


@pytest.fixture(scope="module")
def ctx():
    c = loom_b200.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("batch,K,N", [(1, 32, 1), (2, 64, SLOT // 2 - 1), (2, 64, SLOT // 2), (2, 64, SLOT // 2 + 1), (1, SLOT + 1, 16),
                                       (40, 16400, 64), (40, 64, 16400)])
def test_rows_cross_whole(ctx, batch, K, N):
    rng = np.random.default_rng(K + N)
    m = orc.Matrix.from_f32((rng.standard_normal(N * K) * 0.02).astype(np.float32), N, K)
    w = ctx.upload_ternary(m.words, N, K, m.scale)
    x = torch.from_numpy(rng.standard_normal((batch, K)).astype(np.float32))
    epre, epost = orc.dense_forward(m, cabi.ACT_RELU2, x.numpy())
    for pin_in, pin_out in ((False, False), (True, False), (False, True), (True, True)):
        a = x.clone().pin_memory() if pin_in else x.clone()
        pre, post = (torch.full((batch, N), 7.0, pin_memory=pin_out) for _ in range(2))
        for want_pre, want_post in ((True, True), (True, False), (False, True)):
            pre.fill_(7.0), post.fill_(7.0)
            ctx._check(cabi.lib().loom_b200_dense_forward(ctx.h, w.h, cabi.ACT_RELU2, a.data_ptr(), batch, pre.data_ptr() if want_pre else None,
                                                          post.data_ptr() if want_post else None))
            if want_pre:
                assert (pre.numpy().view(np.uint32) == epre.view(np.uint32)).all()
            if want_post:
                assert (post.numpy().view(np.uint32) == epost.view(np.uint32)).all()


def test_threads_and_contexts_share_the_slots():
    wrong, meet = [], threading.Barrier(7)

    def work(i):
        try:
            rng = np.random.default_rng(i)
            m = orc.Matrix.from_f32((rng.standard_normal(640 * 900) * 0.02).astype(np.float32), 640, 900)
            x = rng.standard_normal((30, 900)).astype(np.float32)
            _, want = orc.dense_forward(m, cabi.ACT_RELU2, x)
            meet.wait(60)
            for _ in range(4):
                c = loom_b200.Context(0)
                w = c.upload_ternary(m.words, 640, 900, m.scale)
                for n in (30, 1, 7):
                    _, post = cabi.dense_forward(c, w, cabi.ACT_RELU2, x[:n])
                    if not np.array_equal(post.view(np.uint32), want[:n].view(np.uint32)):
                        wrong.append((i, n))
                w.free()
                c.close()
        except Exception as e:  # noqa: BLE001 (reported by the caller)
            wrong.append((i, e))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(7)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
