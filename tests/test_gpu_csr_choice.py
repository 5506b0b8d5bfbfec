"""Which kernel the CSR products run on, seen from their sums.

FP64: every row is made of pairs (a, -fl(a x_j)) in neighbouring columns with x = (x_j, 1): the
row-stream kernel rounds each product and adds a pair within a lane, so y is 0 to the last bit; the
CSR kernel fuses multiply and add, so some rows keep a rounding error.  FP32 / BF16 with FP32 sums
(rows of (2^30, 1, -2^30, 0) with x = 1): the row-stream kernel loses the 1, the CSR kernel sums in
FP64."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

ROWS, CSR = "row-stream", "csr"


def _structure(lens, ncols=None):
    """Rows of consecutive columns from an even one on (lens: multiples of 4), along the diagonal."""
    l = torch.as_tensor(lens, dtype=torch.int64).cuda()
    n = l.numel()
    m = ncols or max(n, int(l.max()) + 2)
    row = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    row[1:] = torch.cumsum(l, 0)
    r = torch.repeat_interleave(torch.arange(n, device="cuda"), l)
    e = torch.arange(int(row[-1]), device="cuda") - row[r]
    first = torch.arange(n, device="cuda") * m // n
    first = torch.minimum(first, m - l) // 2 * 2
    return row.int(), (first[r] + e), e, m


def _pairs(lens, ncols=None):
    row, col, e, m = _structure(lens, ncols)
    g = torch.Generator(device="cuda").manual_seed(5)
    x = torch.rand(m, dtype=torch.float64, device="cuda", generator=g)
    x[1::2] = 1.0
    val = torch.randn(col.numel(), dtype=torch.float64, device="cuda", generator=g)
    odd = e % 2 == 1
    val[odd] = -(val[~odd] * x[col[~odd]])
    return row, col.int(), val, x


def kernel_f64(y):
    return ROWS if not y.any() else CSR


def product(lens, fmt=dict(fmt="CSR")):
    from gpu_spmv_b200 import engine as E

    row, col, val, x = _pairs(lens)
    A = E.Matrix(row, col, val, ncols=x.numel(), **fmt)
    y = A.spmv(x)
    A.close()
    return kernel_f64(y)


def arrays(lens):
    from gpu_spmv_b200 import engine as E

    return kernel_f64(E.csr_spmv_f64(*_pairs(lens)))


def dropin(lens):
    from gpu_spmv_b200 import _lib as L
    from gpu_spmv_b200 import refapi as R

    row, col, val, x = (t.cpu().numpy() for t in _pairs(lens, len(lens)))
    h = R.csr_struct(row.view(np.uint32), col.view(np.uint32), val)
    zero = np.zeros(len(lens))
    old = L.lib().gs_get_num_ite()
    L.lib().gs_set_num_ite(2)
    res = L.lib().test_gcsr(256, h.s, R.f64p(x), R.f64p(zero))
    L.lib().gs_set_num_ite(old)
    assert res.name == b"gcsr"
    return kernel_f64(R.last_y(len(lens)))


def reduced(lens, vtype, itype):
    from gpu_spmv_b200 import engine as E

    row, col, e, m = _structure(lens)
    val = torch.tensor([2.0 ** 30, 1.0, -2.0 ** 30, 0.0], device="cuda")[e % 4]
    A = E.Matrix(row, col.int(), val, ncols=m, fmt="CSR", vtype=vtype, itype=itype)
    y = A.spmv(torch.ones(m, device="cuda"))
    A.close()
    n = torch.as_tensor(lens).cuda() / 4
    assert not y.any() or torch.equal(y, n.float())
    return ROWS if not y.any() else CSR


# rows that do not fit a window of 480 positions (FP64) or 1024 together with three others: from
# 6,000 of them on; longer than it: from 20,000
FEW = [(1000, 100, CSR), (300, 300, ROWS), (1000, 200, ROWS), (5999, 200, ROWS), (6000, 200, CSR),
       (30, 10000, ROWS), (19999, 600, ROWS), (20000, 600, CSR)]


@pytest.mark.parametrize("n, length, want", FEW)
def test_few_long_rows(n, length, want):
    lens = [length] * n
    assert product(lens) == want
    assert product(lens, dict(fmt="AXT", mode="COM", tileH=1)) == want
    if length <= n:
        assert dropin(lens) == want


@pytest.mark.parametrize("vtype, itype", [("f32", "u32"), ("f32", "u16"), ("bf16", "u32"),
                                          ("bf16", "u16")])
@pytest.mark.parametrize("n, length, want", [(1000, 200, CSR), (300, 400, ROWS), (5999, 400, ROWS),
                                             (6000, 400, CSR), (30, 10000, ROWS)])
def test_few_long_rows_reduced(vtype, itype, n, length, want):
    assert reduced([length] * n, vtype, itype) == want


def _with(n, length, at):
    """n rows of `length`, but for at = {row: (rows, length)}."""
    lens = [length] * n
    for r, (rows, l) in at.items():
        lens[r:r + rows] = [l] * rows
    return lens


# long rows side by side, which one warp of the CSR kernel would walk one after the other; long rows
# alone or apart, which either kernel gives to one warp
SIDE = {
    "16 of 500": (_with(20000, 28, {9000: (16, 500)}), ROWS),
    "last 8 of 2000": (_with(20000, 28, {19992: (8, 2000)}), ROWS),
    "two apart": (_with(20000, 28, {40: (1, 1000), 17000: (1, 1000)}), CSR),
    "one": (_with(20000, 28, {19999: (1, 12000)}), CSR),
    "one among short ones": (_with(300000, 4, {299999: (1, 30000)}), CSR),
    "128 of 300": (_with(300000, 4, {150016: (128, 300)}), ROWS),
    "64 of 40": (_with(1000, 8, {480: (64, 40)}), ROWS),
    "64 of 40 in many": (_with(3000000, 4, {480: (64, 40)}), CSR),
    "none": ([28] * 20000, CSR),
}


@pytest.mark.parametrize("name", SIDE)
def test_long_rows_side_by_side(name):
    lens, want = SIDE[name]
    assert product(lens) == want
    assert product(lens, dict(fmt="AXT", mode="COM", tileH=1)) == want
    assert dropin(lens) == want


@pytest.mark.parametrize("vtype, itype", [("f32", "u32"), ("bf16", "u16")])
@pytest.mark.parametrize("name, want", [("16 of 500", ROWS), ("one", CSR), ("none", CSR),
                                        ("64 of 40", ROWS)])
def test_long_rows_side_by_side_reduced(vtype, itype, name, want):
    assert reduced(SIDE[name][0], vtype, itype) == want


# rows of 4.5 elements at least, or of 2.5 and nearly all the same; of the FP64 ones 2.5
SHORT = {
    "1 on average": ([4, 0, 0, 0] * 20000, ROWS, ROWS),
    "4": ([4] * 50000, CSR, CSR),
    "4 and none": ([4, 4, 0, 4] * 20000, CSR, ROWS),
    "8 and none": ([8, 0, 8, 0] * 20000, CSR, ROWS),
    "4 and 8": ([4, 8] * 20000, CSR, CSR),
}


@pytest.mark.parametrize("name", SHORT)
def test_short_rows(name):
    lens, f64, other = SHORT[name]
    if max(lens) > 4:  # a pair or two leave no rounding error in either kernel
        assert product(lens) == f64
    for vtype, itype in [("f32", "u32"), ("f32", "u16"), ("bf16", "u32"), ("bf16", "u16")]:
        assert reduced(lens, vtype, itype) == other


# straight from CSR arrays nothing is known of the rows beforehand: a warp that meets more than 49152
# elements beside its longest row leaves them, and the call goes to the row-stream kernel
@pytest.mark.parametrize("name, lens, want", [
    ("16 of 2000", _with(20000, 28, {19984: (16, 2000)}), CSR),
    ("16 of 4000", _with(20000, 28, {19984: (16, 4000)}), CSR),  # 31.2 on average: 8 rows a warp
    ("16 of 8000", _with(20000, 28, {19984: (16, 8000)}), ROWS),
    ("300 of 300", [300] * 300, CSR),
    ("30 of 10000", [10000] * 30, CSR),
    ("30 of 12000", [12000] * 30, CSR),
    ("30 of 20000", [20000] * 30, ROWS),
    ("first 2 of 40000", _with(60000, 28, {0: (2, 40000)}), CSR),
    ("first 2 of 60000", _with(60000, 28, {0: (2, 59998)}), ROWS),
    ("one", _with(100000, 28, {99999: (1, 90000)}), CSR),
    ("two apart", _with(100000, 28, {5: (1, 60000), 99999: (1, 90000)}), CSR),
    ("one among short ones", _with(700000, 4, {699999: (1, 60000)}), CSR),
    ("2 among short ones", _with(700000, 4, {699998: (2, 60000)}), ROWS),
])
def test_arrays_long_rows(name, lens, want):
    for _ in range(2):
        assert arrays(lens) == want


def test_uneven_rows_of_local_columns():
    """FP64 rows of very uneven length, 8 or more elements on average: the row-stream kernel with 8
    positions per lane; y against the exact sums, 1e-13 (|A||x|)_i."""
    from gpu_spmv_b200 import engine as E

    rng = np.random.default_rng(9)
    lens = np.minimum(np.exp(2.0 + 1.5 * rng.standard_normal(300000)), 2000).astype(int) // 4 * 4
    assert lens.mean() >= 8 and product(lens.tolist()) == ROWS
    row, col, e, m = _structure(lens)
    val = torch.randn(col.numel(), dtype=torch.float64, device="cuda")
    x = torch.rand(m, dtype=torch.float64, device="cuda") - 0.5
    A = E.Matrix(row, col.int(), val, ncols=m, fmt="CSR")
    assert A.info.lane_positions == 8
    y = A.spmv(x).cpu().numpy()
    A.close()
    p = (val.cpu().numpy().astype(np.longdouble) * x[col].cpu().numpy().astype(np.longdouble))
    some, at = lens > 0, row.cpu().numpy()[:-1][lens > 0]
    want, mag = np.zeros(len(lens), np.longdouble), np.zeros(len(lens), np.longdouble)
    want[some], mag[some] = np.add.reduceat(p, at), np.add.reduceat(np.abs(p), at)
    assert np.all(np.abs(y - want) <= 1e-13 * mag)
