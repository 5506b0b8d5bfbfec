"""The engine's performance cases: the work that its users have it do, over the sizes they have it
do it at, through the public entry points (``engine.Matrix``, ``engine.csr_spmv_f64``,
``engine.Batch``, ``autograd``).

Each kind of case is one way of using the engine:

``spmv``      repeated products with one converted matrix (an iterative solver, a time loop): the
              matrix is converted beforehand, a pass is one product;
``csr``       one product straight from CSR arrays that are assembled anew every time;
``convert``   a new matrix: its conversion to a format and its first product;
``spmm``      a product with several right-hand sides at once;
``gradient``  one training step of a layer with sparse weights: the step's new values go in, the
              forward product, then the gradients of the operand and of the values;
``operator``  the gradients of a matrix seen for the first time (sensitivities of a newly assembled
              system): an operator is built and run forward and backward once through autograd;
``batch``     many uneven banded systems, each with its own right-hand sides, in one launch.

Ranges.  Laplacians of 64^2 to 2048^2 grid points, 27-point stencils of 16^3 to 160^3, power-law
matrices of 4 Ki to 4 Mi rows with 16 elements a row on average (lognormal lengths), banded
matrices of 1,000 to 200,000 rows with half-bandwidths 16 to 256 and 5 to 60 elements a row; FP64,
FP32 and BF16 values, 32- and 16-bit columns; 1 to 32 right-hand sides.

Matrices are made on the GPU with torch from the seed alone.  A matrix's element count follows from
its case, not from the seed.
"""
from __future__ import annotations

import math
import random

import torch

from gpu_spmv_b200 import autograd as AG
from gpu_spmv_b200 import engine as E

DTYPE = {"f64": torch.float64, "f32": torch.float32, "bf16": torch.float32}  # operands
VBYTES = {"f64": 8, "f32": 4, "bf16": 2}  # stored values


# ---------------------------------------------------------------------------------- matrices
def _rng(seed: int, stream: int) -> torch.Generator:
    g = torch.Generator(device="cuda")
    g.manual_seed(1000003 * int(seed) + stream)
    return g


def _row_ptr(lens: torch.Tensor) -> torch.Tensor:
    row = torch.zeros(lens.numel() + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(lens, 0, out=row[1:])
    return row


def _laplacian(grid: int, seed: int):
    """5-point Laplacian of a grid x grid mesh: 4 on the diagonal, -1 beside it."""
    n = grid * grid
    p = torch.arange(n, device="cuda")
    i, j = p // grid, p % grid
    off = torch.tensor([-grid, -1, 0, 1, grid], device="cuda")
    keep = torch.stack([i > 0, j > 0, i >= 0, j < grid - 1, i < grid - 1], 1)
    col = (p[:, None] + off)[keep]
    val = torch.where(off == 0, 4.0, -1.0).double().expand(n, 5)[keep]
    return _row_ptr(keep.sum(1)), col, val


def _stencil(grid: int, seed: int):
    """27-point stencil on grid^3: 26 on the diagonal, -1 + U(-0.1, 0.1) beside it."""
    n = grid ** 3
    p = torch.arange(n, device="cuda")
    z, y, x = p // (grid * grid), (p // grid) % grid, p % grid
    d = torch.tensor([-1, 0, 1], device="cuda")
    dz, dy, dx = (t.reshape(-1) for t in torch.meshgrid(d, d, d, indexing="ij"))
    keep = torch.ones(n, 27, dtype=torch.bool, device="cuda")
    for c, dc in ((z, dz), (y, dy), (x, dx)):
        q = c[:, None] + dc
        keep &= (q >= 0) & (q < grid)
    off = (dz * grid + dy) * grid + dx
    col = (p[:, None] + off)[keep]
    diag = (off == 0).expand(n, 27)[keep]
    val = -1.1 + 0.2 * torch.rand(col.numel(), generator=_rng(seed, 1), device="cuda",
                                  dtype=torch.float64)
    val[diag] = 26.0
    return _row_ptr(keep.sum(1)), col, val


def _powerlaw(rows: int, seed: int):
    """Lognormal(2.5, 1.2) row lengths clipped to [1, 10000] and rescaled to 16 a row on average;
    columns uniform, ascending in a row; values N(0, 1)."""
    g = _rng(seed, 2)
    nnz = 16 * rows
    raw = torch.exp(2.5 + 1.2 * torch.randn(rows, generator=g, device="cuda",
                                            dtype=torch.float64)).clamp(1, 10000)
    lens = (raw * (nnz / raw.sum())).floor().clamp(1, max(1, rows // 4)).long()
    perm = torch.randperm(rows, generator=g, device="cuda")
    left = nnz - int(lens.sum())
    while left:  # the rounding, spread over rows at random
        cand = perm if left > 0 else perm[lens[perm] > 1]
        take = cand[:abs(left)]
        lens[take] += 1 if left > 0 else -1
        left -= take.numel() if left > 0 else -take.numel()
    key = torch.repeat_interleave(torch.arange(rows, device="cuda"), lens)
    key = key * rows + torch.randint(rows, (nnz,), generator=g, device="cuda")
    col = torch.sort(key).values.remainder_(rows)
    del key
    val = torch.randn(nnz, generator=g, device="cuda", dtype=torch.float64)
    return _row_ptr(lens), col, val


def _banded(rows: int, half: int, seed: int):
    """5 to 60 elements a row inside the band, one in each of as many equal parts of it; values
    N(0, 1)."""
    g = _rng(seed, 3)
    lo = (torch.arange(rows, device="cuda") - half).clamp(min=0)
    hi = (torch.arange(rows, device="cuda") + half + 1).clamp(max=rows)
    lens = _banded_lens(rows, half)[torch.randperm(rows, generator=g, device="cuda")]
    row = _row_ptr(lens)
    r = torch.repeat_interleave(torch.arange(rows, device="cuda"), lens)
    j = torch.arange(r.numel(), device="cuda") - row[r]
    w, m = (hi - lo)[r], lens[r]
    a, b = j * w // m, (j + 1) * w // m
    u = torch.rand(r.numel(), generator=g, device="cuda", dtype=torch.float64)
    col = lo[r] + a + ((b - a) * u).long()
    val = torch.randn(r.numel(), generator=g, device="cuda", dtype=torch.float64)
    return row, col, val


def _banded_lens(rows: int, half: int) -> torch.Tensor:
    top = min(60, half + 1)  # a corner row has half + 1 columns in its band
    return 5 + torch.arange(rows, device="cuda") % (top - 4)


def _csr(case: dict, seed: int):
    """(row int32 bits of u32, col, val) of the case's matrix on the GPU."""
    m, size = case["matrix"], case["size"]
    if m == "laplacian":
        row, col, val = _laplacian(size, seed)
    elif m == "stencil":
        row, col, val = _stencil(size, seed)
    elif m == "powerlaw":
        row, col, val = _powerlaw(size, seed)
    else:
        row, col, val = _banded(size, case["half"], seed)
    vt = case.get("vtype", "f64")
    if vt == "f32":
        val = val.float()
    elif vt == "bf16":  # weights that were saved in BF16
        val = val.bfloat16().float()
    return row.int(), col.int(), val


def _shape(case: dict):
    """(rows, elements) of the case's square matrix."""
    m, s = case["matrix"], case["size"]
    if m == "laplacian":
        return s * s, 5 * s * s - 4 * s
    if m == "stencil":
        return s ** 3, (3 * s - 2) ** 3
    if m == "powerlaw":
        return s, 16 * s
    return s, _banded_nnz(s, case["half"])


def _banded_nnz(rows: int, half: int) -> int:
    span = min(60, half + 1) - 4
    full, rest = divmod(rows, span)
    return 5 * rows + full * (span * (span - 1) // 2) + rest * (rest - 1) // 2


def _dense(n: int, k: int, dtype, seed: int, stream: int) -> torch.Tensor:
    shape = (n,) if k == 0 else (n, k)
    return torch.randn(*shape, generator=_rng(seed, stream), device="cuda",
                       dtype=torch.float64).to(dtype)


def _x(case: dict, n: int, seed: int) -> torch.Tensor:
    """Single operands: uniform on [-1, 1)."""
    u = torch.rand(n, generator=_rng(seed, 10), device="cuda", dtype=torch.float64)
    return (2 * u - 1).to(DTYPE[case.get("vtype", "f64")])


# ---------------------------------------------------------------------------------- the cases
def listed():
    return [
        # the smallest products, where a launch and the host's part of a call count: the 5-point
        # Laplacian that solvers are tried on first
        dict(name="spmv_laplacian_csr", kind="spmv", matrix="laplacian", size=512, fmt="CSR",
             vtype="f64"),
        # the largest product, in the format that general matrices are converted to
        dict(name="spmv_powerlaw_k1", kind="spmv", matrix="powerlaw", size=4194304, fmt="K1",
             vtype="f64"),
        # the same matrix family in tiles, a ragged number of rows
        dict(name="spmv_powerlaw_axt4", kind="spmv", matrix="powerlaw", size=2999999, fmt="AXT",
             mode="UNC", tileH=4, vtype="f64"),
        # a 3D discretisation in reduced storage: FP32 values with 16-bit column steps
        dict(name="spmv_stencil_f32", kind="spmv", matrix="stencil", size=160, fmt="K1",
             vtype="f32", itype="u16"),
        # the smallest storage the engine has, with FP64 sums, on an odd grid
        dict(name="spmv_stencil_bf16", kind="spmv", matrix="stencil", size=131, fmt="CSR",
             vtype="bf16", itype="u16", acc64=True),
        # a matrix assembled anew for every product (its values change, its CSR arrays are all
        # there is)
        dict(name="csr_stencil", kind="csr", matrix="stencil", size=101),
        # a new matrix: conversion and first product
        dict(name="convert_powerlaw_k1", kind="convert", matrix="powerlaw", size=1048576,
             fmt="K1", vtype="f64"),
        # block Krylov and feature propagation: eight right-hand sides
        dict(name="spmm_powerlaw_f32_k8", kind="spmm", matrix="powerlaw", size=1048576,
             vtype="f32", k=8),
        # a block solver with an odd number of right-hand sides left
        dict(name="spmm_banded_f64_k5", kind="spmm", matrix="banded", size=199999, half=200,
             vtype="f64", k=5),
        # a training step: new values, forward, both gradients
        dict(name="gradient_powerlaw_f32_k8", kind="gradient", matrix="powerlaw", size=1048576,
             vtype="f32", k=8, mode="deterministic"),
        # first gradients of a newly assembled system
        dict(name="operator_powerlaw_f64_k3", kind="operator", matrix="powerlaw", size=262143,
             vtype="f64", k=3),
        # many uneven systems in one launch
        dict(name="batch_banded_f32", kind="batch", count=64, mix=3, vtype="f32"),
    ]


def _log(rng: random.Random, lo: float, hi: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_matrix(rng: random.Random, kinds, top: float = 1.0) -> dict:
    """A matrix of the ranges above; `top` scales the upper ends down by elements."""
    m = rng.choice(kinds)
    if m == "laplacian":
        return dict(matrix=m, size=_log(rng, 64, 2048 * top ** 0.5))
    if m == "stencil":
        return dict(matrix=m, size=_log(rng, 16, 160 * top ** (1 / 3)))
    if m == "powerlaw":
        return dict(matrix=m, size=_log(rng, 4096, 4194304 * top))
    return dict(matrix=m, size=_log(rng, 1000, 200000), half=rng.randint(16, 256))


FORMATS = [dict(fmt="CSR"), dict(fmt="K1"), dict(fmt="AXC"), dict(fmt="AXT", mode="COM", tileH=1),
           dict(fmt="AXT", mode="COM", tileH=4), dict(fmt="AXT", mode="UNC", tileH=1),
           dict(fmt="AXT", mode="UNC", tileH=2), dict(fmt="AXT", mode="UNC", tileH=4),
           dict(fmt="AXT", mode="UNC", tileH=8)]
ALL = ("laplacian", "stencil", "powerlaw", "banded")


def draw(rng: random.Random) -> dict:
    kind = rng.choice(["spmv", "spmv", "reduced", "csr", "convert", "spmm", "gradient", "operator",
                       "batch"])
    if kind == "spmv":
        return dict(kind="spmv", vtype="f64", **_draw_matrix(rng, ALL), **rng.choice(FORMATS))
    if kind == "reduced":
        m = _draw_matrix(rng, ALL)
        local = m["matrix"] != "powerlaw"  # 16-bit steps need a row's columns close together
        return dict(kind="spmv", vtype=rng.choice(["f32", "bf16"]), fmt=rng.choice(["CSR", "K1"]),
                    itype=rng.choice(["u32", "u16"]) if local else "u32",
                    acc64=rng.choice([False, True]), **m)
    if kind == "csr":
        return dict(kind="csr", **_draw_matrix(rng, ALL, 0.25))
    if kind == "convert":
        return dict(kind="convert", vtype=rng.choice(["f64", "f64", "f32"]),
                    fmt=rng.choice(["CSR", "K1"]), **_draw_matrix(rng, ALL, 0.25))
    if kind == "spmm":
        return dict(kind="spmm", vtype=rng.choice(["f32", "f64"]), k=rng.randint(1, 16),
                    **_draw_matrix(rng, ALL, 0.125))
    if kind == "gradient":
        return dict(kind="gradient", vtype=rng.choice(["f32", "f64"]), k=rng.randint(1, 16),
                    mode=rng.choice(["deterministic", "deterministic", "atomic"]),
                    **_draw_matrix(rng, ALL, 0.125))
    if kind == "operator":
        return dict(kind="operator", vtype=rng.choice(["f32", "f64"]), k=rng.randint(1, 8),
                    **_draw_matrix(rng, ALL, 0.0625))
    return dict(kind="batch", count=rng.randint(8, 64), mix=rng.randint(0, 1 << 20),
                vtype=rng.choice(["f32", "f32", "f64"]))


def _members(case: dict):
    """The matrices of a batch: rows log-uniform in [1000, 200000], half-bandwidth 16 to 256, 1 to
    32 right-hand sides."""
    rng = random.Random(case["mix"])
    return [dict(matrix="banded", size=_log(rng, 1000, 200000), half=rng.randint(16, 256),
                 vtype=case["vtype"], k=rng.randint(1, 32)) for _ in range(case["count"])]


def _convert(case: dict, row, col, val):
    keys = ("fmt", "mode", "tileH", "vtype", "itype")
    return E.Matrix(row, col, val, **{k: case[k] for k in keys if k in case})


# ---------------------------------------------------------------------------------- a pass
def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    st = {"case": case}
    if kind == "batch":
        st["mats"], Xs = [], []
        for i, m in enumerate(_members(case)):
            row, col, val = _csr(m, 4096 * seed + i)
            st["mats"].append(E.Matrix(row, col, val, fmt="K1", vtype=case["vtype"]))
            Xs.append(_dense(m["size"], m["k"], DTYPE[case["vtype"]], 4096 * seed + i, 11))
        st["batch"] = E.Batch(st["mats"], [m["k"] for m in _members(case)])
        st["batch"].make_operands(Xs)
        return st
    row, col, val = _csr(case, seed)
    n = row.numel() - 1
    if kind == "spmv":
        st["A"] = _convert(case, row, col, val)
        st["x"] = _x(case, n, seed)
        return st
    if kind in ("csr", "convert"):
        st.update(row=row, col=col, val=val, x=_x(case, n, seed))
        return st
    dt, k = DTYPE[case["vtype"]], case["k"]
    st["X"] = _dense(n, k, dt, seed, 11)
    if kind == "spmm":
        st["A"] = E.Matrix(row, col, val, fmt="K1", vtype=case["vtype"])
        return st
    st["Ybar"] = _dense(n, k, dt, seed, 12)  # the gradient that the rest of the model hands back
    if kind == "gradient":
        st["A"] = E.Matrix(row, col, val, fmt="K1", vtype=case["vtype"], adjoint=True)
        st["v"] = _dense(col.numel(), 0, dt, seed, 13)  # the step's values
        return st
    st.update(row=row, col=col, val=val)
    return st


def run(st: dict):
    case = st["case"]
    kind = case["kind"]
    if kind == "spmv":
        return st["A"].spmv(st["x"], acc64=case.get("acc64", False))
    if kind == "csr":
        return E.csr_spmv_f64(st["row"], st["col"], st["val"], st["x"])
    if kind == "convert":
        return _convert(case, st["row"], st["col"], st["val"]).spmv(st["x"])
    if kind == "spmm":
        return st["A"].spmm(st["X"])
    if kind == "gradient":
        A = st["A"]
        A.set_values(st["v"])
        Y = A.spmm(st["X"])
        Xbar, vbar = A.adjoint(st["Ybar"], st["X"], mode=case["mode"])
        return Y, Xbar, vbar
    if kind == "operator":
        op = AG.SparseOperator(st["row"], st["col"], st["val"], vtype=case["vtype"])
        v = st["val"].detach().requires_grad_()
        X = st["X"].detach().requires_grad_()
        Y = AG.spmm(v, X, op)
        vbar, Xbar = torch.autograd.grad(Y, (v, X), st["Ybar"])
        return Y.detach(), Xbar, vbar
    st["batch"].run()
    return st["batch"].results()


# ---------------------------------------------------------------------------------- what it needs
def _product_work(n: int, nnz: int, k: int, vb: int, ib: int, xb: int, yb: int):
    return nnz * (vb + ib) + 4 * (n + 1) + (xb + yb) * n * k, 2 * nnz * k


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "batch":
        b = f = 0
        vb = VBYTES[case["vtype"]]
        for m in _members(case):
            mb, mf = _product_work(*_shape(m), m["k"], vb, 4, vb, vb)
            b, f = b + mb, f + mf
        return {"bytes": b, "flops": f}
    n, nnz = _shape(case)
    vt = case.get("vtype", "f64")
    vb, ib = VBYTES[vt], 2 if case.get("itype") == "u16" else 4
    xb = 8 if vt == "f64" else 4
    yb = 8 if case.get("acc64") else xb
    k = case.get("k", 1)
    if kind == "convert":
        vb = xb  # the values as they come
    b, f = _product_work(n, nnz, k, vb, ib, xb, yb)
    if kind in ("gradient", "operator"):
        # the matrix once, X and Ybar in, Y, Xbar and the value gradient out
        b = nnz * (2 * vb + ib) + 4 * (n + 1) + 4 * xb * n * k
        f = 6 * nnz * k
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------------------------- in 64 bits
def _exact_mm(row, col, val, X):
    n = row.numel() - 1
    A = torch.sparse_csr_tensor(row.long(), col.long(), val.double(), (n, n))
    return A @ X.double()


def _exact_gradients(row, col, X, Ybar, val):
    n, nnz = row.numel() - 1, col.numel()
    c = col.long()
    r = torch.repeat_interleave(torch.arange(n, device="cuda"), row.long().diff())
    X64, Y64 = X.double(), Ybar.double()
    vbar = torch.empty(nnz, dtype=torch.float64, device="cuda")
    for a in range(0, nnz, 1 << 22):
        s = slice(a, a + (1 << 22))
        vbar[s] = (Y64[r[s]] * X64[c[s]]).sum(1)
    order = torch.argsort(c, stable=True)
    ptr = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(torch.bincount(c, minlength=n), 0, out=ptr[1:])
    AT = torch.sparse_csr_tensor(ptr, r[order], val.double()[order], (n, n))
    return AT @ Y64, vbar


def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind == "batch":
        out = []
        for i, m in enumerate(_members(case)):
            row, col, val = _csr(m, 4096 * seed + i)
            X = _dense(m["size"], m["k"], DTYPE[case["vtype"]], 4096 * seed + i, 11)
            out.append(_exact_mm(row, col, val, X))
        return out
    row, col, val = _csr(case, seed)
    n = row.numel() - 1
    if kind in ("spmv", "csr", "convert"):
        return _exact_mm(row, col, val, _x(case, n, seed))
    dt, k = DTYPE[case["vtype"]], case["k"]
    X = _dense(n, k, dt, seed, 11)
    if kind == "spmm":
        return _exact_mm(row, col, val, X)
    if kind == "gradient":
        val = _dense(col.numel(), 0, dt, seed, 13)
    Xbar, vbar = _exact_gradients(row, col, X, _dense(n, k, dt, seed, 12), val)
    return _exact_mm(row, col, val, X), Xbar, vbar
