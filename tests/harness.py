"""tests/kernel_harness.cu, compiled by nvcc against the library's own headers and linked with it."""
import ctypes as C
import functools
import os
import subprocess
import tempfile

from loom_b200 import build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@functools.lru_cache(None)
def lib():
    lb, out = build.LIB, os.path.join(tempfile.mkdtemp(), "kernel_harness.so")
    flags = [f for f in build.NVCC_FLAGS if f not in ("-Xptxas", "-v")]
    subprocess.run([build.nvcc(), *flags, "-shared", "-I", os.path.join(ROOT, "include"), "-I", build.CSRC, os.path.join(ROOT, "tests", "kernel_harness.cu"), lb,
                    "-Xlinker", "-rpath," + os.path.dirname(lb), "-o", out], check=True)
    so = C.CDLL(out)
    vp, i, f = C.c_void_p, C.c_int, C.c_float
    so.t_gemm_bf16.argtypes = [vp, i, vp, vp, vp, i, vp, i, vp, i, i, i, f, f, f]
    so.t_attention_prompt.argtypes = [vp, vp, vp, vp, vp, vp, i, i, i, i, i]
    so.t_pair_begin.argtypes = [vp, C.POINTER(vp)]
    so.t_pair_message.argtypes = [vp, C.c_uint, i, vp, vp, vp, i]
    so.t_pair_end.argtypes = [vp, vp]
    so.t_pair_end.restype = None
    return so
