"""A process that resets its device goes on with a new context under the same device number: the library's calls work in it
as in the first.  The process is a child that talks to the library and the runtime alone (torch does not survive a reset)."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import ctypes, importlib.util, sys
import numpy as np
spec = importlib.util.spec_from_file_location("jq_lib", sys.argv[1])
jq = importlib.util.module_from_spec(spec)
spec.loader.exec_module(jq)
lib, rt = jq.load(), ctypes.CDLL("libcudart.so.12")
rt.cudaMalloc.argtypes = [ctypes.c_void_p, ctypes.c_size_t]
rt.cudaMemcpy.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_size_t, ctypes.c_int]
N, K, T = 256, 2048, 64
rng = np.random.default_rng(1)
qw = rng.integers(0, 256, (N, K // 2), dtype=np.uint8)
cb = np.sort(rng.standard_normal((N, 16))).astype(np.float16)
sc = rng.uniform(0.5, 1, (N, K // 32)).astype(np.float16)
x = rng.standard_normal((T, K)).astype(np.float32)
img = rng.standard_normal((1, 32, 8, 8)).astype(np.float32)      # 2048 = 32 channels x 8 x 8: kernels of 8 x 8
def ok(st):
    assert st == 0, jq.strerror(st) if st < 0 else st
def device(a=None, nbytes=0):
    p = ctypes.c_void_p()
    ok(rt.cudaMalloc(ctypes.byref(p), a.nbytes if a is not None else nbytes))
    src = a if a is not None else np.zeros(nbytes, np.uint8)
    ok(rt.cudaMemcpy(p, src.ctypes.data, src.nbytes, 1))
    return p
def everything():
    dq, dc, ds, dx, di = (device(a) for a in (qw, cb, sc, x, img))
    y, ws, status = device(nbytes=T * N * 4), device(nbytes=8 << 20), device(nbytes=256)
    outs = []
    def out(rows):
        h = np.empty((rows, N), np.float32)
        ok(rt.cudaMemcpy(h.ctypes.data, y, h.nbytes, 2))
        outs.append(h)
    for fmt, scales, g, B in ((1, ds, 128, 1), (1, ds, 128, 8), (1, ds, 128, 24), (1, ds, 128, 64), (0, ds, 32, 16), (0, ds, 32, 40)):
        ok(lib.jq_gemm_ta(fmt, dq, scales, dc, dx, None, y, N, K, B, g, 0, 0, 0, ws, 8 << 20, None))
        out(B)
        assert lib.jq_ta_status(ws, 0, None) == 0
    for fmt, g in ((1, 128), (0, 32), (0, 64)):
        ok(lib.jq_gemm_rows(fmt, dq, ds, dc, dx, None, y, N, K, T, g, 0, 0, 0, ws, 8 << 20, status, None))
        out(T)
    for k, pad in ((8, 0), (8, 3)):
        side = 8 + 2 * pad - k + 1
        c = jq.jq_conv(1, 32, 8, 8, k, k, 1, 1, pad, pad, 1, 1, (ctypes.c_int64 * 4)(2048, 64, 8, 1))
        ok(lib.jq_conv_rows(1, dq, ds, dc, di, None, y, ctypes.byref(c), N, K, side * side, 128, 0, 0, ws, 8 << 20, status, None))
        out(side * side)
    c = jq.jq_conv(1, 32, 8, 8, 4, 4, 1, 1, 0, 0, 1, 1, (ctypes.c_int64 * 4)(2048, 64, 8, 1))     # fields kept in shared memory
    ok(lib.jq_conv_rows(1, dq, ds, dc, di, None, y, ctypes.byref(c), N, 512, 25, 128, 0, 0, ws, 8 << 20, status, None))
    out(25)
    return outs
first = everything()
ok(rt.cudaDeviceReset())
for a, b in zip(first, everything()):
    assert np.isfinite(a).all() and np.abs(a).max() > 0 and np.array_equal(a, b)
print("same")
"""


def test_calls_after_the_device_was_reset():
    lib = os.path.join(ROOT, "if_i_could_turn_back_time_b200", "_lib.py")
    r = subprocess.run([sys.executable, "-c", CHILD, lib], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "same", r.stderr[-2000:]


NO_ALLOC = CHILD[:CHILD.index("N, K, T = ")] + r"""
N, K, B = 96, 28672, 8             # more activation than fits in shared memory: partial sums in the library's own array
rng = np.random.default_rng(2)
qw = rng.integers(0, 256, (N, K // 2), dtype=np.uint8)
sc = rng.uniform(0.5, 1, (N, K // 32)).astype(np.float16)
x = rng.standard_normal((B, K)).astype(np.float32)
def ok(st):
    assert st == 0, jq.strerror(st) if st < 0 else st
def device(a):
    p = ctypes.c_void_p()
    ok(rt.cudaMalloc(ctypes.byref(p), a.nbytes))
    ok(rt.cudaMemcpy(p, a.ctypes.data, a.nbytes, 1))
    return p
def call():
    y = np.zeros((B, N), np.float32)
    dy = device(y)
    ok(lib.jq_gemv_noalloc(0, device(qw), device(sc), None, device(x), None, dy, N, K, B, 32, 0, 0, 0, None))
    ok(rt.cudaMemcpy(y.ctypes.data, dy, y.nbytes, 2))
    return y
first = [call(), call()]
ok(rt.cudaDeviceReset())
device(np.zeros(64 << 20, np.uint8))      # (the new context's memory is laid out otherwise)
for y in first + [call(), call()]:
    assert np.isfinite(y).all() and np.abs(y).max() > 0 and np.array_equal(y, first[0])
print("same")
"""


def test_calls_without_workspace_after_the_device_was_reset():
    """The array of the allocation-free entry is looked up again: its address in the first context means nothing in the next."""
    lib = os.path.join(ROOT, "if_i_could_turn_back_time_b200", "_lib.py")
    r = subprocess.run([sys.executable, "-c", NO_ALLOC, lib], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "same", r.stderr[-2000:]
