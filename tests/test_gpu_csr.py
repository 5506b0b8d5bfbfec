"""The CSR kernel (CSR and COM tileH = 1 of local columns and even rows, the product straight from CSR arrays)
where its windows of 256, 512 and 1024 positions can go wrong: rows and groups of 32 rows that end
at, before and after a window's end, groups of empty rows, rows over many windows, few long rows
among short ones (several lanes per row), the streams' ends, and arrays that are 16- but not
32-byte aligned; every stored type and column width.

FP64: 1e-13 (|A||x|)_i.  FP32 / BF16: the products are rounded to FP32, the sums are FP64 and y is
rounded once, so |err_i| <= 2^-24 (|A||x|)_i + 2^-24 |y_i| plus FP64 terms."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

E31 = [0] * 31
LENS = {
    "one": [1],
    "empty": [0] * 70,
    "short": [5] * 3001,
    "full256": [8] * 64 + [7] * 31 + [8 * 32 - 7 * 31] + [8] * 33,
    "full512": [16] * 96 + [0] * 31 + [512] + [15] * 32,
    "full1024": [32] * 96 + [0] * 31 + [1024] + [0] * 31 + [1025] + [31] * 40,
    "stencil": [27] * 999,
    "runs": (E31 + [3] + E31 * 3 + [300] + [0, 0, 1]) * 9 + E31 * 5,
    "long": [0, 40000, 0, 0, 7, 0],
    "uneven": [1, 200, 3, 90, 2, 2, 31, 32, 33, 64, 500, 0] * 50,
    "pow2": [64] * 64 + [128] * 40,
}


def _even(lens):
    """`lens` and as many rows of their average length as make them even (32 times the longest of
    each 32 rows at most 2.5 times the elements): what gs_matrix_create sends to this kernel."""
    avg = max(1, round(sum(lens) / len(lens)))
    waste = sum(32 * max(lens[i:i + 32]) for i in range(0, len(lens), 32)) - 2.5 * sum(lens)
    return lens + [avg] * (32 * max(0, int(waste / (32 * 1.5 * avg)) + 2)) if sum(lens) else lens


def _csr(lens, seed, local=True):
    """Columns of a row ascend by 1 to 8 (one run where the row is long) or at random, within 60000
    columns (16-bit columns fit)."""
    rng = np.random.default_rng(seed)
    lens = np.asarray(lens)
    row = np.zeros(len(lens) + 1, np.uint32)
    row[1:] = np.cumsum(lens)
    cols = [np.zeros(0, int)]
    for l in lens:
        if local:
            c = np.cumsum(rng.integers(1, 9 if l < 5000 else 2, l))
            cols.append(c + rng.integers(0, 60000 - (c[-1] if l else 0)))
        else:
            cols.append(np.sort(rng.choice(60000, l, replace=False)))
    col = np.concatenate(cols).astype(np.uint32)
    return row, col, rng.standard_normal(len(col))


def _exact(row, col, val, x):
    p = val * x[col]
    s = lambda a: np.array([np.sum(a[b:e]) for b, e in zip(row[:-1], row[1:])])
    return s(p), s(np.abs(p))


@pytest.mark.parametrize("name", LENS)
@pytest.mark.parametrize("fmt", [dict(fmt="CSR"), dict(fmt="AXT", mode="COM", tileH=1)],
                         ids=["csr", "com1"])
def test_f64(name, fmt):
    from gpu_spmv_b200 import engine as E

    row, col, val = _csr(_even(LENS[name]), 3)
    x = np.random.default_rng(4).uniform(-1, 1, 60000)
    want, mag = _exact(row, col, val, x)
    A = E.Matrix(row, col, val, ncols=60000, **fmt)
    xd = torch.from_numpy(x).cuda()
    y = torch.full((len(want),), float("nan"), dtype=torch.float64, device="cuda")
    A.spmv(xd, y)
    assert np.all(np.abs(y.cpu().numpy() - want) <= 1e-13 * mag)
    assert torch.equal(y, A.spmv(xd))
    A.close()


@pytest.mark.parametrize("name", LENS)
@pytest.mark.parametrize("off", [0, 4])
@pytest.mark.parametrize("local", [True, False])
def test_csr_arrays(name, off, local):
    """gs_csr_spmv_f64 on exact-size arrays that start 0 or 16 bytes past a 256-byte boundary."""
    from gpu_spmv_b200 import engine as E

    row, col, val = _csr(LENS[name], 5, local)
    x = np.random.default_rng(6).uniform(-1, 1, 60000)
    want, mag = _exact(row, col, val, x)
    dev = torch.device("cuda")
    d_col = torch.zeros(len(col) + off, dtype=torch.int32, device=dev)[off:]
    d_val = torch.zeros(len(val) + off // 2, dtype=torch.float64, device=dev)[off // 2:]
    d_col.copy_(E.to_device_u32(col, dev))
    d_val.copy_(torch.from_numpy(val))
    y = E.csr_spmv_f64(E.to_device_u32(row, dev), d_col, d_val, torch.from_numpy(x).cuda())
    assert np.all(np.abs(y.cpu().numpy() - want) <= 1e-13 * mag)


@pytest.mark.parametrize("name", LENS)
@pytest.mark.parametrize("vtype", ["f32", "bf16"])
@pytest.mark.parametrize("itype", ["u32", "u16"])
@pytest.mark.parametrize("acc64", [False, True])
def test_reduced(name, vtype, itype, acc64):
    from gpu_spmv_b200 import engine as E

    row, col, val = _csr(_even(LENS[name]), 7)
    t = torch.from_numpy(val)
    val = (t.bfloat16() if vtype == "bf16" else t.float()).double().numpy()
    x = np.random.default_rng(8).uniform(-1, 1, 60000).astype(np.float32)
    want, mag = _exact(row, col, val, x.astype(np.float64))
    A = E.Matrix(row, col, val, ncols=60000, fmt="CSR", vtype=vtype, itype=itype)
    y = A.spmv(torch.from_numpy(x).cuda(), acc64=acc64)
    assert y.dtype == (torch.float64 if acc64 else torch.float32)
    bound = 2.0 ** -24 * mag * (1 + 1e-6) + (0 if acc64 else 2.0 ** -24 * np.abs(want) * (1 + 1e-6))
    assert np.all(np.abs(y.double().cpu().numpy() - want) <= bound)
    A.close()
