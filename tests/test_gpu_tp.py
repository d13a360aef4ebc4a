"""Tensor parallelism on the GPU.  The one-GPU cases run the row-sharded path with a group of one (no exchange,
but the supplied-statistics prologue, the raw-accumulator epilogue and the finalize kernel) and as rank 0 of a pair whose second rank is
played by messages that lie in the mailbox beforehand; the multi-GPU case
needs at least two GPUs and runs one process per GPU against the unsharded CPU oracle."""
import ctypes as C
import os
import socket
import subprocess
import sys

import numpy as np
import pytest

import harness
from loom_b200 import cabi
from oracle import oracle as orc
from refkit import np_unpack

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


def free_port() -> int:
    with socket.socket() as s:
        s.bind(("127.0.0.1", 0))
        return s.getsockname()[1]


@pytest.mark.parametrize("rows,K,batch,with_inner", [(96, 256, 1, True), (2560, 6912, 1, False), (130, 1040, 8, True)])
def test_rowsharded_linear_group_of_one(rows, K, batch, with_inner):
    ctx = cabi.Context(0)
    ctx.tp_init(0, 1, bytes(128))
    assert ctx.tp_world == 1 and ctx.tp_rank == 0
    rng = np.random.default_rng(rows + K)
    words, scale = orc.pack_f32((rng.standard_normal(rows * K) * 0.05).astype(np.float32), rows, K)
    inner = (1 + 0.1 * rng.standard_normal(K)).astype(np.float32) if with_inner else None
    bias = (0.01 * rng.standard_normal(rows)).astype(np.float32)
    x = rng.standard_normal((batch, K)).astype(np.float32)
    w = ctx.upload_ternary(words, rows, K, scale)
    d_x, d_b = ctx.to_device(x), ctx.to_device(bias)
    d_in = ctx.to_device(inner) if with_inner else None
    d_out = ctx.alloc(batch * rows * 4)
    ctx.tp_rowsharded_linear(w, batch, d_x, K, d_out, inner_w=d_in, inner_w_len=K if with_inner else 0, eps=0.0, bias=d_b)
    got = ctx.download(d_out, (batch, rows), np.float32)
    for t in range(batch):
        xq, amax = orc.quantize_f32(orc.inner_rmsnorm_f32(x[t], inner, 0.0))
        acc = orc.matvec_i32(words, rows, K, xq).astype(np.float64)
        want = (acc * float(np.float64(scale) * np.float64(amax) / 127.0) + bias.astype(np.float64)).astype(np.float32)
        assert np.array_equal(got[t], want)
    with pytest.raises(cabi.LoomB200Error):
        ctx.tp_rowsharded_linear(w, 9, d_x, K, d_out)  # more tokens than one pass carries
    with pytest.raises(cabi.LoomB200Error):
        ctx.tp_rowsharded_linear(w, 1, d_x, K - 16, d_out)  # whole vector narrower than the slice
    ctx.close()


@pytest.mark.parametrize("fused", [0, 1])
def test_rowsharded_linear_of_rank_0_of_two(fused):
    """Three and eight tokens through the peer exchange on one GPU: the second rank's sums lie in the mailbox before the first rank asks for
    them.  Twice each, behind narrower and wider shards on one context; bit for bit."""
    ctx = cabi.Context(0)
    other = C.c_void_p()
    ctx._check(harness.lib().t_pair_begin(ctx.h, C.byref(other)))
    ctx.set_option("tp_fused", fused)
    seq = 0
    try:
        for rows, Kl, batch in ((96, 256, 3), (96, 256, 8), (2560, 4096, 8), (130, 1040, 3), (300, 4096, 5), (96, 256, 8), (64, 640, 1)):
            rng = np.random.default_rng(rows + Kl + batch)
            K = 2 * Kl
            full = (rng.standard_normal((rows, K)) * 0.05).astype(np.float32)
            words, scale = orc.pack_f32(full.reshape(-1), rows, K)
            codes = np_unpack(words, rows, K)
            shard = np.ascontiguousarray(words.reshape(rows, -1)[:, :Kl // 16])
            w = ctx.upload_ternary(shard, rows, Kl, scale)
            inner, bias = (1 + 0.1 * rng.standard_normal(K)).astype(np.float32), (0.01 * rng.standard_normal(rows)).astype(np.float32)
            d_in, d_b, d_out = ctx.to_device(inner[:Kl]), ctx.to_device(bias), ctx.alloc(batch * rows * 4)
            for _ in range(2):
                seq += 1
                x = rng.standard_normal((batch, K)).astype(np.float32)
                y = np.stack([orc.inner_rmsnorm_f32(r, inner, 0.0) for r in x])
                q, amax = orc.quantize_rows_f32(y)
                acc = q.astype(np.int32) @ codes.astype(np.int32).T
                theirs = np.ascontiguousarray(q[:, Kl:].astype(np.int32) @ codes[:, Kl:].astype(np.int32).T)
                ss, top = (x[:, Kl:].astype(np.float64) ** 2).sum(1), np.ascontiguousarray(np.abs(y[:, Kl:]).max(1))
                ctx._check(harness.lib().t_pair_message(ctx.h, seq, batch, ss.ctypes.data, top.ctypes.data, theirs.ctypes.data, theirs.size))
                d_x = ctx.to_device(np.ascontiguousarray(x[:, :Kl]))
                ctx.tp_rowsharded_linear(w, batch, d_x, K, d_out, inner_w=d_in, inner_w_len=Kl, eps=0.0, bias=d_b)
                got = ctx.download(d_out, (batch, rows), np.float32)
                ctx.sync()
                # (a pass of more tokens than a group's passes carry)
                q20, a20 = orc.quantize_rows_f32(rng.standard_normal((20, Kl)).astype(np.float32))
                d20 = [ctx.to_device(q20), ctx.to_device(a20), ctx.alloc(20 * rows * 4)]
                ctx.ternary_linear(w, 20, d20[0], d20[1], None, acc_out=d20[2])
                assert np.array_equal(ctx.download(d20[2], (20, rows), np.int32), q20.astype(np.int32) @ codes[:, :Kl].astype(np.int32).T)
                for p in d20:
                    ctx.free(p)
                want = (acc * (np.float64(scale) * amax.astype(np.float64) / 127.0)[:, None] + bias.astype(np.float64)).astype(np.float32)
                assert np.array_equal(got, want)
                ctx.free(d_x)
            for p in (d_in, d_b, d_out):
                ctx.free(p)
    finally:
        harness.lib().t_pair_end(ctx.h, other)
        ctx.close()


def test_decoder_refuses_dimensions_that_do_not_divide():
    # a group of one accepts everything; the divisibility rule itself is covered on the CPU by the shard plan
    ctx = cabi.Context(0)
    dec = cabi.Decoder(ctx, 1, 64, 4, 1, 16, 96, 50, 1e-5, 10000.0)
    dec.close()
    ctx.close()


@pytest.mark.parametrize("mode", ["nograph", "graph", "peer", "peer3"])
def test_two_ranks_match_unsharded_oracle(mode):
    import torch
    if torch.cuda.device_count() < 2:
        pytest.skip("needs two GPUs")
    env = dict(os.environ)
    env.update(OMP_NUM_THREADS="4", NCCL_NVLS_ENABLE="0")
    cmd = [sys.executable, "-m", "torch.distributed.run", "--nnodes=1", "--nproc-per-node", "2", "--master-addr", "127.0.0.1",
           "--master-port", str(free_port()), os.path.join(HERE, "tp_gpu_worker.py"), mode]
    r = subprocess.run(cmd, env=env, capture_output=True, text=True, timeout=420)
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr[-3000:]
    assert "rank 0 ok" in r.stdout and "rank 1 ok" in r.stdout
