"""Kernels in a second context of the process, which stands for a second device: what one context was told (how much shared memory a
kernel may have) does not hold in another."""
from __future__ import annotations

import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

CHILD = r"""
import ctypes
import numpy as np
from thintensor_b200.kernels import build

cuda = ctypes.CDLL("libcuda.so.1")


def check(code):
    assert code == 0, f"driver call failed: {code}"


def on_device(array):
    at = ctypes.c_uint64()
    check(cuda.cuMemAlloc_v2(ctypes.byref(at), ctypes.c_size_t(array.nbytes)))
    check(cuda.cuMemcpyHtoD_v2(at, array.ctypes.data_as(ctypes.c_void_p), ctypes.c_size_t(array.nbytes)))
    return at.value


def product_in_parts():
    m, n, k = 40, 300, 200
    rng = np.random.default_rng(0)
    x, w = rng.standard_normal((m, k), dtype=np.float32), rng.standard_normal((n, k), dtype=np.float32)
    out, status = np.zeros((m, n), np.float32), np.zeros(1, np.int32)
    px, pw, po, ps, parts = on_device(x), on_device(w), on_device(out), on_device(status), on_device(np.zeros((3, m, k), np.uint16))
    fn = build.load("gemm_split").tt_gemm_split
    p, i, l = ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong
    fn.argtypes, fn.restype = [p, l, p, l, p, p, l, l, p, p, i, i, i, i, i, p], i
    code = fn(px, k, pw, k, None, po, n, m * n, parts, ps, m, n, k, 1, 148, None)
    assert code == 0, f"the launch failed: {code}"
    check(cuda.cuCtxSynchronize())
    check(cuda.cuMemcpyDtoH_v2(out.ctypes.data_as(p), ctypes.c_uint64(po), ctypes.c_size_t(out.nbytes)))
    want = x.astype(np.float64) @ w.astype(np.float64).T
    assert np.abs(out - want).max() < 1e-4, np.abs(out - want).max()


def bfloat16_product():
    m, n, k = 40, 256, 128
    rng = np.random.default_rng(1)
    # numbers that bfloat16 holds, and sums that float32 holds
    x, w = rng.integers(-4, 5, (m, k)).astype(np.float32), rng.integers(-4, 5, (n, k)).astype(np.float32)
    narrow = lambda a: (a.view(np.uint32) >> 16).astype(np.uint16)
    out, status = np.zeros((m, n), np.float32), np.zeros(1, np.int32)
    px, pw, po, ps = on_device(narrow(x)), on_device(narrow(w)), on_device(out), on_device(status)
    fn = build.load("gemm_tcgen05").tt_gemm_tcgen05
    p, i, l = ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong
    fn.argtypes, fn.restype = [p, l, p, l, p, p, l, l, i, i, i, i, i, p, p, p, l], i
    code = fn(px, k, pw, k, None, po, n, m * n, m, n, k, 1, 0, ps, None, None, 0)
    assert code == 0, f"the launch failed: {code}"
    check(cuda.cuCtxSynchronize())
    check(cuda.cuMemcpyDtoH_v2(out.ctypes.data_as(p), ctypes.c_uint64(po), ctypes.c_size_t(out.nbytes)))
    assert np.array_equal(out, x @ w.T)


check(cuda.cuInit(0))
device = ctypes.c_int()
check(cuda.cuDeviceGet(ctypes.byref(device), 0))
first, second = ctypes.c_void_p(), ctypes.c_void_p()
check(cuda.cuDevicePrimaryCtxRetain(ctypes.byref(first), device))
check(cuda.cuCtxSetCurrent(first))
product_in_parts()
bfloat16_product()
check(cuda.cuCtxCreate_v2(ctypes.byref(second), ctypes.c_uint(0), device))
check(cuda.cuCtxSetCurrent(second))
product_in_parts()
bfloat16_product()
print("both contexts")
"""


def test_products_in_a_second_context():
    done = subprocess.run([sys.executable, "-c", CHILD], cwd=Path(__file__).resolve().parent.parent, capture_output=True, text=True, timeout=300)
    assert done.returncode == 0 and "both contexts" in done.stdout, done.stdout + done.stderr
