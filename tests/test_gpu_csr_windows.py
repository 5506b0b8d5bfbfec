"""The CSR kernel where its windows end: a warp's rows (4 to 128) that end one position before, at and
one after the end of their window (288, 480 or 1024 positions, counted from the multiple of 8 at or
before their first element), with their elements spread, in the first, in the last or in both, from
every start within 8 positions; rows of several windows; groups of empty rows; a last group that is
not full; plain and padded windows (rows of about 8 m elements); every stored type and column width.

FP64: 1e-13 (|A||x|)_i.  FP32 / BF16 with FP64 y: products rounded to FP32 and summed in FP64, so
|err_i| <= 2^-24 (|A||x|)_i plus FP64 terms; with FP32 y the same sums, rounded once, which only this
kernel gives."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

COLS = 60000


def _shape(n, nnz, f64):
    """Window, rows per warp and padding that the launch chooses."""
    big, avg = (480 if f64 else 1024), nnz / n
    fits = lambda rows, cap: avg * rows <= (cap - 8) / 1.05
    pad = round(avg) > 0 and round(avg) % 8 == 0 and abs(avg - round(avg)) < 0.5
    if fits(64, 480) and n // 64 >= 148 * 32:
        return 480, 128 if fits(128, 480) and n // 128 >= 148 * 32 else 64, pad
    if fits(32, 288):
        return 288, 32, pad
    if fits(32, 480):
        return 480, 32, pad
    for rows in (32, 16, 8):
        if fits(rows, big):
            return big, rows, pad
    return big, 4, pad


def _group(total, rows, how):
    lens = np.zeros(rows, np.int64)
    if how == "spread":
        lens[:] = total // rows
        lens[:total % rows] += 1
    elif how == "ends":
        lens[0], lens[-1] = total // 2, total - total // 2
    else:
        lens[0 if how == "first" else -1] = total
    return lens


def _spread(lens):
    """32 times the longest row of each 32 over the elements."""
    full = lens[:len(lens) // 32 * 32].reshape(-1, 32)
    return 32 * full.max(1).sum() / full.sum()


def _lens(cap, rows, avg, groups, tail, even=0.0):
    """Groups of `rows` rows that reach cap - 1, cap, cap + 1 from each start mod 8, each behind a
    group that brings its start about and keeps the average; a long row, an empty group; ordinary
    groups of `avg` a row, up to `groups` and until the rows are as even as `even` (with 1.25, no
    longest rows either); `tail` rows."""
    out, pos = [], 0
    flat = 0 < even < 2

    def add(lens):
        nonlocal pos
        out.append(lens)
        pos += int(lens.sum())

    ordinary = int(round(avg * rows))
    for how in ("spread",) if flat else ("spread", "first", "last", "ends"):
        for d in (-1, 0, 1):
            for start in range(8):
                fill = 2 * ordinary - (cap + d - start)
                add(_group(fill + (start - pos - fill) % 8, rows, "spread"))
                assert pos % 8 == start
                add(_group(cap + d - start, rows, how))
    if not flat:
        long = np.zeros(rows, np.int64)
        long[rows // 2] = 2 * cap + 5
        add(long)
        add(np.zeros(rows, np.int64))
        add(_group(2 * ordinary, rows, "spread"))
    while len(out) < groups or even and _spread(np.concatenate(out)) > 0.95 * even:
        for _ in range(50):
            add(_group(ordinary, rows, "spread"))
    out.append(np.full(tail, int(round(avg)), np.int64))
    return np.concatenate(out)


def _matrix(lens, seed):
    rng = np.random.default_rng(seed)
    row = np.zeros(len(lens) + 1, np.int64)
    np.cumsum(lens, out=row[1:])
    step = np.cumsum(rng.integers(1, 9, row[-1]))
    r = np.repeat(np.arange(len(lens)), lens)
    col = step - step[row[r]]
    last = np.zeros(len(lens), np.int64)
    last[lens > 0] = col[row[1:][lens > 0] - 1]
    col += rng.integers(0, COLS - last)[r]
    return row.astype(np.uint32), col.astype(np.uint32), rng.standard_normal(len(col))


def _exact(row, col, val, x):
    p = val.astype(np.longdouble) * x[col].astype(np.longdouble)
    some = np.diff(row.astype(np.int64)) > 0
    y, mag = np.zeros(len(some), np.longdouble), np.zeros(len(some), np.longdouble)
    y[some] = np.add.reduceat(p, row[:-1][some].astype(np.int64))
    mag[some] = np.add.reduceat(np.abs(p), row[:-1][some].astype(np.int64))
    return y.astype(np.float64), mag.astype(np.float64)


# window, rows per warp, average row, padded, groups
F64 = [(288, 32, 7, False, 400), (288, 32, 8, True, 400), (480, 32, 12, False, 400),
       (480, 32, 8.38, True, 400), (480, 16, 20, False, 400), (480, 16, 24, True, 400),
       (480, 8, 44, False, 400), (480, 8, 48, True, 400), (480, 4, 100, False, 400),
       (480, 4, 104, True, 400), (480, 64, 5, False, 4737), (480, 128, 3, False, 4737),
       (480, 64, 7, False, 4737), (288, 32, 5, False, 9400)]
REDUCED = [s for s in F64 if s[1] >= 32] + [
    (1024, 32, 20, False, 400), (1024, 32, 24, True, 400), (1024, 16, 44, False, 400),
    (1024, 16, 48, True, 400), (1024, 8, 100, False, 400), (1024, 8, 104, True, 400),
    (1024, 4, 200, False, 400), (1024, 4, 207, True, 400)]


def _ids(shapes):
    return [f"{s[0]}x{s[1]}{'pad' if s[3] else ''}-{s[2]}" for s in shapes]


@pytest.mark.parametrize("tail", [0, 1, 3])
@pytest.mark.parametrize("shape", F64, ids=_ids(F64))
def test_f64(shape, tail):
    from gpu_spmv_b200 import engine as E

    cap, rows, avg, pad, groups = shape
    lens = _lens(cap, rows, avg, groups, tail)
    assert _shape(len(lens), int(lens.sum()), True) == (cap, rows, pad)
    row, col, val = _matrix(lens, rows)
    x = np.random.default_rng(1).uniform(-1, 1, COLS)
    want, mag = _exact(row, col, val, x)
    dev = torch.device("cuda")
    y = torch.full((len(lens),), float("nan"), dtype=torch.float64, device=dev)
    E.csr_spmv_f64(E.to_device_u32(row, dev), E.to_device_u32(col, dev),
                   torch.from_numpy(val).cuda(), torch.from_numpy(x).cuda(), y)
    assert np.all(np.abs(y.cpu().numpy() - want) <= 1e-13 * mag)


@pytest.mark.parametrize("vtype, itype", [("f32", "u32"), ("f32", "u16"), ("bf16", "u32"),
                                          ("bf16", "u16")])
@pytest.mark.parametrize("shape", REDUCED, ids=_ids(REDUCED))
def test_reduced(vtype, itype, shape):
    from gpu_spmv_b200 import engine as E

    cap, rows, avg, pad, groups = shape
    lens = _lens(cap, rows, avg, groups, 3, 1.25 if avg < 4.5 else 2.5)
    assert _shape(len(lens), int(lens.sum()), False) == (cap, rows, pad)
    row, col, val = _matrix(lens, rows + 1)
    t = torch.from_numpy(val)
    val = (t.bfloat16() if vtype == "bf16" else t.float()).double().numpy()
    x = np.random.default_rng(2).uniform(-1, 1, COLS).astype(np.float32)
    want, mag = _exact(row, col, val, x.astype(np.float64))
    A = E.Matrix(row, col, val, ncols=COLS, fmt="CSR", vtype=vtype, itype=itype)
    xd = torch.from_numpy(x).cuda()
    y = A.spmv(xd, acc64=True)
    assert torch.equal(A.spmv(xd), y.float())
    assert np.all(np.abs(y.cpu().numpy() - want) <= 2.0 ** -24 * mag * (1 + 1e-6))
    A.close()
