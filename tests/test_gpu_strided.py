"""Multi-RHS products and the adjoint for any number of right-hand sides and any row strides: every
column equals the single-RHS K1 product bit for bit (the same sums in the same order), for A and,
as the adjoint, for the explicit transpose, with rows over several work pieces; the value gradient
against its definition, |err| <= (k + 1) eps sum |Ybar||X|."""
import numpy as np
import pytest
import torch

from mats import csr_from_lengths

pytestmark = pytest.mark.gpu


def _matrix(seed):
    rng = np.random.default_rng(seed)
    lens = rng.integers(0, 30, 1000)
    lens[7], lens[500] = 700, 300  # cut chunks
    row, col, val = csr_from_lengths(lens, 900, rng)
    col = np.where(rng.random(len(col)) < 0.2, 5, col).astype(np.uint32)  # a long column
    return row, col, val


def _transpose(row, col, val, ncols):
    order = np.argsort(col, kind="stable")
    rows = np.repeat(np.arange(len(row) - 1), np.diff(row))
    row_t = np.concatenate([[0], np.cumsum(np.bincount(col, minlength=ncols))]).astype(np.uint32)
    return row_t, rows[order].astype(np.uint32), val[order]


def _operand(rng, n, k, dt, how):
    """[n, k]: contiguous; columns 3 .. of a wider array; every second row; transposed."""
    full = torch.from_numpy(rng.standard_normal((2 * n, k + 7))).to(dt).cuda()
    if how == "tight":
        return full[:n, :k].contiguous()
    if how == "columns":
        return full[:n, 3:3 + k]
    if how == "rows":
        return full[::2, :k]
    return full[:n, :k].t().contiguous().t()


@pytest.mark.parametrize("vtype", ["f64", "f32"])
@pytest.mark.parametrize("k", [1, 2, 3, 4, 5, 6, 7, 8, 9, 12, 15, 16, 17, 20, 24, 30, 31, 32, 40])
@pytest.mark.parametrize("how", ["tight", "columns", "rows", "transposed"])
def test_any_width(vtype, k, how):
    from gpu_spmv_b200 import engine as E

    rng = np.random.default_rng(k)
    row, col, val = _matrix(3)
    dt = torch.float64 if vtype == "f64" else torch.float32
    A = E.Matrix(row, col, val, ncols=900, fmt="K1", vtype=vtype, adjoint=True)
    T = E.Matrix(*_transpose(row, col, val, 900), ncols=1000, fmt="K1", vtype=vtype)
    X, Yb = _operand(rng, 900, k, dt, how), _operand(rng, 1000, k, dt, how)
    Y = A.spmm(X)
    Xbar, vbar = A.adjoint(Yb, X)
    Xonly, none = A.adjoint(Yb, want_vbar=False)
    assert none is None and torch.equal(Xbar, Xonly)
    for c in range(k):
        assert torch.equal(Y[:, c], A.spmv(X[:, c].contiguous()))
        assert torch.equal(Xbar[:, c], T.spmv(Yb[:, c].contiguous()))
    r = np.repeat(np.arange(1000), np.diff(row))
    y, x = Yb.double().cpu().numpy()[r], X.double().cpu().numpy()[col]
    want, mag = np.einsum("ek,ek->e", y, x), np.einsum("ek,ek->e", np.abs(y), np.abs(x))
    eps = 2.0 ** -53 if vtype == "f64" else 2.0 ** -24
    err = np.abs(vbar.double().cpu().numpy() - want)
    assert np.all(err <= ((k + 1) * eps + k * 2.0 ** -52) * mag)
    A.close()
    T.close()


def test_refusals():
    from gpu_spmv_b200 import _lib as L
    from gpu_spmv_b200 import engine as E

    row, col, val = _matrix(4)
    A = E.Matrix(row, col, val, ncols=900, fmt="K1")
    X, Y = torch.zeros(900, 40, device="cuda").double(), torch.zeros(1000, 40, device="cuda").double()
    f = L.lib().gs_spmm_strided
    assert f(A._h, X.data_ptr(), 40, Y.data_ptr(), 40, L.GS_F64, 33, 40, None) == L.GS_ERR_UNSUPPORTED
    assert f(A._h, X.data_ptr(), 40, Y.data_ptr(), 40, L.GS_F64, 0, 40, None) == L.GS_ERR_UNSUPPORTED
    assert f(A._h, X.data_ptr(), 4, Y.data_ptr(), 40, L.GS_F64, 5, 5, None) == L.GS_ERR_INVALID
    assert f(A._h, X.data_ptr() + 4, 40, Y.data_ptr(), 40, L.GS_F64, 5, 5, None) == L.GS_ERR_INVALID
    assert f(A._h, X.data_ptr(), 40, Y.data_ptr(), 40, L.GS_F32, 5, 5, None) == L.GS_ERR_UNSUPPORTED
    assert f(A._h, X.data_ptr(), 40, Y.data_ptr(), 40, L.GS_F64, 5, 4, None) == L.GS_ERR_INVALID
    assert f(A._h, X.data_ptr(), 6, Y.data_ptr(), 40, L.GS_F64, 5, 8, None) == L.GS_ERR_INVALID
    assert L.lib().gs_spmm(A._h, X.data_ptr(), Y.data_ptr(), L.GS_F64, 5, None) == L.GS_ERR_UNSUPPORTED
    A.close()


@pytest.mark.parametrize("k", [3, 4, 5, 8, 40])
def test_adjoint_operand_forms(k):
    """Row counts that fit neither the matrix nor a broadcast are refused on the host; a single
    column or row is broadcast and a host tensor moved where the product copies its operands."""
    from gpu_spmv_b200 import engine as E

    rng = np.random.default_rng(k)
    row, col, val = _matrix(5)
    A = E.Matrix(row, col, val, ncols=900, fmt="K1", adjoint=True)
    X = _operand(rng, 900, k, torch.float64, "columns")
    Yb = _operand(rng, 1000, k, torch.float64, "columns")
    Xbar, vbar = A.adjoint(Yb, X)
    for bad_y, bad_x in [(Yb[:-1], X), (Yb, X[:-1]), (torch.cat([Yb, Yb[:1]]), X[:-1])]:
        with pytest.raises(RuntimeError):
            A.adjoint(bad_y, bad_x)
        with pytest.raises(RuntimeError):
            A.adjoint(bad_y.contiguous(), bad_x.contiguous())
    same = A.adjoint(Yb, X.cpu())
    assert torch.equal(same[0], Xbar) and torch.equal(same[1], vbar)
    assert torch.equal(A.adjoint(Yb.contiguous(), X.float())[1],
                       A.adjoint(Yb, X.float().double())[1])
    assert torch.equal(A.adjoint(Yb, X[:1])[1], A.adjoint(Yb, X[:1].expand(900, k).contiguous())[1])
    with pytest.raises(TypeError):
        A.spmm(X[:-1])
    A.close()


@pytest.mark.parametrize("vtype", ["f64", "f32"])
def test_value_gradient_orders_32(vtype):
    """32 right-hand sides: the CSR-order value gradient is the slot-order one, moved (every entry
    written), also beside an Xbar of its own."""
    from gpu_spmv_b200 import engine as E

    rng = np.random.default_rng(32)
    row, col, val = _matrix(6)
    dt = torch.float64 if vtype == "f64" else torch.float32
    A = E.Matrix(row, col, val, ncols=900, fmt="K1", vtype=vtype, adjoint=True)
    X, Yb = _operand(rng, 900, 32, dt, "tight"), _operand(rng, 1000, 32, dt, "tight")
    for _ in range(2):
        Xc, vc = A.adjoint(Yb, X)
        Xs, vs = A.adjoint(Yb, X, order="slots")
        assert torch.equal(vc, A.convert_values(vs, to="csr")) and torch.equal(Xc, Xs)
        assert torch.equal(vs, A.convert_values(vc, to="slots"))
    A.close()


def test_adjoint_refusals():
    from gpu_spmv_b200 import _lib as L
    from gpu_spmv_b200 import engine as E

    row, col, val = _matrix(4)
    A = E.Matrix(row, col, val, ncols=900, fmt="K1", adjoint=True)
    B = E.Matrix(row, col, val, ncols=900, fmt="K1")
    C = E.Matrix(row, col, val, ncols=900, fmt="CSR")
    X, Xb = (torch.zeros(900, 40, device="cuda").double() for _ in range(2))
    Yb, v = torch.zeros(1000, 40, device="cuda").double(), torch.zeros(len(col)).double().cuda()
    x, xb, yb, vb = X.data_ptr(), Xb.data_ptr(), Yb.data_ptr(), v.data_ptr()
    bad, no = L.GS_ERR_INVALID, L.GS_ERR_UNSUPPORTED
    for want, m, args in [
            (no, A, (yb, 40, x, 40, xb, 40, vb, L.GS_F64, 33, 40)),
            (no, A, (yb, 40, x, 40, xb, 40, vb, L.GS_F64, 0, 40)),
            (no, A, (yb, 40, x, 40, xb, 40, vb, L.GS_F32, 5, 5)),
            (no, C, (yb, 40, x, 40, xb, 40, vb, L.GS_F64, 5, 5)),
            (bad, B, (yb, 40, x, 40, xb, 40, vb, L.GS_F64, 5, 5)),     # no adjoint prepared
            (bad, A, (yb, 40, x, 40, xb, 40, vb, L.GS_F64, 5, 4)),     # fewer columns than k
            (bad, A, (yb, 6, x, 40, xb, 40, vb, L.GS_F64, 5, 8)),      # readable past a row
            (bad, A, (yb, 40, x, 6, xb, 40, vb, L.GS_F64, 5, 8)),
            (bad, A, (yb, 40, x, 40, xb, 4, vb, L.GS_F64, 5, 5)),      # rows overlap
            (bad, A, (yb + 4, 40, x, 40, xb, 40, vb, L.GS_F64, 5, 5)),
            (bad, A, (yb, 40, x + 4, 40, xb, 40, vb, L.GS_F64, 5, 5)),
            (bad, A, (yb, 40, x, 40, xb + 4, 40, vb, L.GS_F64, 5, 5)),
            (bad, A, (None, 40, x, 40, xb, 40, vb, L.GS_F64, 5, 5)),
            (bad, A, (yb, 40, None, 40, xb, 40, vb, L.GS_F64, 5, 5)),  # a value gradient needs X
            (bad, A, (yb, 40, x, 40, None, 40, vb, L.GS_F64, 5, 5)),
            (L.GS_OK, A, (yb, 40, None, 0, xb, 40, None, L.GS_F64, 5, 5))]:
        assert L.lib().gs_spmm_adjoint_strided(m._h, *args, None) == want, args
    torch.cuda.synchronize()
    for m in (A, B, C):
        m.close()
