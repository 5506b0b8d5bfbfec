"""The drop-in ncsr, which test_* results are scored against: rows that fit one lane's share (4 or 8
neighbouring elements) equal the CPU loop, product by product and in order, to the last bit.  And
a K1 struct that test_gk1 refuses."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _loop(row, col, val, x):
    y = np.zeros(len(row) - 1)
    for i in range(len(y)):
        s = 0.0
        for e in range(row[i], row[i + 1]):
            s = s + val[e] * x[col[e]]
        y[i] = s
    return y


# length 4: a lane holds 4 elements (short rows); 8: one holds 8 (local columns)
@pytest.mark.parametrize("name", ["ncsr", "gs2_cf_CSR"])
@pytest.mark.parametrize("length", [4, 8])
@pytest.mark.parametrize("n", [1, 31, 3000])
def test_rows_of_a_lane(name, length, n):
    from gpu_spmv_b200 import _lib as L
    from gpu_spmv_b200 import refapi as R

    rng = np.random.default_rng(n)
    cols = max(n, length)
    row = np.arange(n + 1, dtype=np.uint32) * length
    first = np.minimum(np.arange(n), cols - length)
    col = (first[:, None] + np.arange(length)).ravel().astype(np.uint32)
    val = rng.standard_normal(n * length)
    x = rng.uniform(-1, 1, max(n, cols))
    if n < length:  # square matrices: fewer columns than a row's elements, so columns repeat
        col = np.minimum(col, n - 1)
    h = R.csr_struct(row, col, val)
    y = np.full(n, np.nan)
    if name == "ncsr":
        L.lib().ncsr(8, h.s, R.f64p(x), R.f64p(y))
    else:
        g = L.Gen2MatCSR()
        for f in ("nrows", "nnz", "val", "row", "col", "rl"):
            setattr(g, f, getattr(h.s, f))
        L.lib().gs2_cf_CSR(g, R.f64p(x), R.f64p(y))
    assert np.array_equal(y, _loop(row.astype(int), col, val, x))


@pytest.mark.parametrize("chunks", [200, 512])
def test_k1_plan_too_large(chunks):
    """A K1 struct whose steps add up to more work units than 32 bits count is refused before any
    kernel runs on its plan (200 chunks of 2^32 - 1 steps: 6.7e9 units)."""
    from gpu_spmv_b200 import _lib as L
    from gpu_spmv_b200 import refapi as R

    n = chunks * 32
    u32 = lambda a: np.ascontiguousarray(a, np.uint32)
    arrays = dict(permi=u32(np.arange((chunks + 1) * 32) % n), nmc=u32(np.full(chunks, 0xffffffff)),
                  chp=u32(np.arange(chunks) * 32), col=u32(np.zeros(n)))
    val, x = np.zeros(n), np.zeros(n)
    k = L.StrMatK1()
    k.nrows, k.nnz, k.chunkNum, k.lenVC = n, n, chunks, n
    for f, a in arrays.items():
        setattr(k, f, a.ctypes.data_as(L.UINp))
    k.val = val.ctypes.data_as(L.FPTp)
    assert L.lib().test_gk1(256, k, R.f64p(x), R.f64p(x)).name == b"error"
    assert b"K1 plan too large" in L.lib().gs_last_error()
