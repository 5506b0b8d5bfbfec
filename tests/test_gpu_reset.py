"""The library after cudaDeviceReset by the program (its own CUDA runtime, as any caller's): what it
keeps from one call to the next ended with the context, and calls after it work as before.  Runs in
processes of their own, without PyTorch, whose state such a reset ends as well; nothing is in flight
when it comes."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r'''
import ctypes as C, importlib, sys, types
import numpy as np
root, what = sys.argv[1:]
pkg = types.ModuleType("gpu_spmv_b200")  # the bindings alone: the package imports torch
pkg.__path__ = [root + "/gpu_spmv_b200"]
sys.modules["gpu_spmv_b200"] = pkg
L = importlib.import_module("gpu_spmv_b200._lib")
R = importlib.import_module("gpu_spmv_b200.refapi")
assert "torch" not in sys.modules
lib = L.lib()
lib.gs_set_num_ite(2)
rt = C.CDLL("libcudart.so.12")
rng = np.random.default_rng(0)
n = 1000
row = np.arange(n + 1, dtype=np.uint32) * 4
col = np.sort(rng.integers(0, n, (n, 4)), 1).ravel().astype(np.uint32)
val, x = rng.standard_normal(4 * n), rng.uniform(-1, 1, n)
want = (val * x[col]).reshape(n, 4).sum(1)
h = R.csr_struct(row, col, val)

def matrix(fmt):
    p = L.ConvertParams(fmt, 32, 1, 256, L.GS_AXT_COM, 32, L.GS_F64, L.GS_IDX_U32, 0)
    A = C.c_void_p()
    L.check(lib.gs_matrix_create_host(C.byref(A), C.byref(p), n, n, 4 * n, row.ctypes.data,
                                      col.ctypes.data, val.ctypes.data, L.GS_F64, None), "create")
    return A

def dropin():
    y = np.full(n, np.nan)
    lib.ncsr(1, h.s, R.f64p(x), R.f64p(y))
    assert np.abs(y - want).max() <= 1e-13, lib.gs_last_error()
    k = L.StrMatK1()
    assert lib.getFormatDataK1(32, h.s, R.f64p(x), C.byref(k)).name == b"fk1", lib.gs_last_error()
    assert lib.test_gk1(256, k, R.f64p(x), R.f64p(want)).name == b"gk1", lib.gs_last_error()
    assert np.abs(R.last_y(n) - want).max() <= 1e-13

def matrices():
    for fmt in (L.GS_FMT_CSR, L.GS_FMT_K1, L.GS_FMT_AXT):
        A = matrix(fmt)
        y = np.full(n, np.nan)
        L.check(lib.gs_spmv_host_stream(A, x.ctypes.data, 0, L.GS_F64, y.ctypes.data, 0, L.GS_F64,
                                        1, 0, None), "host_stream")
        assert np.abs(y - want).max() <= 1e-13
        lib.gs_matrix_destroy(A)

def held():  # a matrix that outlives the reset is only destroyed
    matrices()
    return matrix(L.GS_FMT_K1)

def batch():
    mats = [matrix(L.GS_FMT_K1) for _ in range(2)]
    dX, dY = [], []
    for i in range(2):
        for arr, d in ((x, dX), (np.zeros(n), dY)):
            p = C.c_void_p()
            assert rt.cudaMalloc(C.byref(p), n * 8) == 0
            assert rt.cudaMemcpy(p, arr.ctypes.data_as(C.c_void_p), n * 8, 1) == 0
            d.append(p.value)
    B = C.c_void_p()
    L.check(lib.gs_batch_create(C.byref(B), 2, (C.c_void_p * 2)(*[m.value for m in mats]),
                                (L.UIN * 2)(1, 1), None), "batch")
    L.check(lib.gs_batch_set_operands(B, (C.c_void_p * 2)(*dX), (C.c_void_p * 2)(*dY), None), "set")
    L.check(lib.gs_batch_run_graph(B, None), "run")
    assert rt.cudaDeviceSynchronize() == 0
    for d in dY:
        y = np.full(n, np.nan)
        L.check(lib.gs_copy_to_host(y.ctypes.data, d, n * 8), "copy")
        assert np.abs(y - want).max() <= 1e-13
    lib.gs_batch_destroy(B)
    for m in mats:
        lib.gs_matrix_destroy(m)

def static():  # the K1 product whose scratch is a device array of the library
    k = L.StrMatK1()
    assert lib.getFormatDataK1(32, h.s, R.f64p(x), C.byref(k)).name == b"fk1", lib.gs_last_error()
    a = R.k1_arrays(k)
    dev = []
    for v in (a["val"], a["col"], a["nmc"], a["chp"], a["permi"], x, np.zeros(n)):
        p = C.c_void_p()
        assert rt.cudaMalloc(C.byref(p), v.nbytes) == 0
        assert rt.cudaMemcpy(p, v.ctypes.data_as(C.c_void_p), v.nbytes, 1) == 0
        dev.append(p.value)
    L.check(lib.gs_k1_spmv_f64_static(n, k.chunkNum, k.lenVC, *dev, None), "static")
    assert rt.cudaDeviceSynchronize() == 0
    y = np.full(n, np.nan)
    L.check(lib.gs_copy_to_host(y.ctypes.data, dev[-1], n * 8), "copy")
    assert np.abs(y - want).max() <= 1e-13

kept = []
for step in range(3):
    kept.append(dict(dropin=dropin, matrices=matrices, held=held, batch=batch,
                     static=static)[what]())
    assert rt.cudaDeviceSynchronize() == 0
    assert rt.cudaDeviceReset() == 0
    if what == "held":
        lib.gs_matrix_destroy(kept[-1])
print("done")
'''


@pytest.mark.parametrize("what", ["dropin", "matrices", "held", "batch", "static"])
def test_after_reset(what):
    r = subprocess.run([sys.executable, "-c", PROGRAM, ROOT, what], capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("done"), r.stdout + r.stderr
