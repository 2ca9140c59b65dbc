"""A C host may reset the device between two calls: its allocations and the context are gone, the library
works on (only fmha_bwd_static_scratch keeps an address of the old context, as the header says)."""
import os
import subprocess
import sys

import pytest

from tests.conftest import PKG

pytestmark = pytest.mark.gpu

# its own process: the reset would take torch's context with it
HOST = """
import ctypes, math, os, sys
lib = ctypes.CDLL(os.path.join(sys.argv[1], "lib", "libfmha_b200.so"))
rt = ctypes.CDLL(os.path.join(os.environ.get("CUDA_HOME") or "/usr/local/cuda", "lib64", "libcudart.so"))
ptr, c_int = ctypes.c_void_p, ctypes.c_int
lib.fmha_b200_forward.argtypes = [ptr] * 5 + [c_int] * 5 + [ctypes.c_float, c_int, ptr]
lib.fmha_b200_backward.argtypes = [ptr] * 10 + [ctypes.c_size_t] + [c_int] * 5 + [ctypes.c_float, c_int, ptr]
rt.cudaMemset.argtypes, rt.cudaMemcpy.argtypes = [ptr, c_int, ctypes.c_size_t], [ptr, ptr, ctypes.c_size_t, c_int]

def zeros(nbytes):
    p = ptr()
    assert rt.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(nbytes)) == 0 and rt.cudaMemset(p, 0, nbytes) == 0
    return p

def both_passes(D, n=256, ws=1 << 22):
    q, k, v, o, do, dq, dk, dv = [zeros(n * D * 2) for _ in range(8)]
    lse, work, host = zeros(n * 4), zeros(ws), (ctypes.c_float * n)()
    assert lib.fmha_b200_forward(q, k, v, o, lse, 1, 1, n, n, D, 0.1, 0, None) == 0
    assert lib.fmha_b200_backward(q, k, v, o, do, lse, dq, dk, dv, work, ws, 1, 1, n, n, D, 0.1, 0, None) == 0
    assert rt.cudaDeviceSynchronize() == 0 and rt.cudaMemcpy(host, lse, n * 4, 2) == 0
    assert all(abs(x - math.log(n)) < 1e-5 for x in host)

for D in (64, 96, 128):
    both_passes(D)
assert rt.cudaDeviceReset() == 0
for D in (64, 96, 128, 64):
    both_passes(D)
"""


def test_calls_after_a_device_reset():
    run = subprocess.run([sys.executable, "-c", HOST, PKG], capture_output=True, text=True, timeout=300)
    assert run.returncode == 0, run.stderr[-2000:]
