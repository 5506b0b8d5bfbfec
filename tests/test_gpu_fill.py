"""K1 slots filled by tiles of 16 steps and pieces of 128: values, columns and padding against numpy
at row lengths around the tiles' and pieces' edges, from arrays at any element offset; new values
put into the same slots; the lane-blocked 16-bit layout through its product.  Equal, not close."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

LENS = {
    "uniform": None,
    "falling": [300, 200, 144, 129, 128, 127, 40, 33, 32, 31, 17, 16, 15, 9, 8, 7, 4, 3, 2, 1, 0] * 4,
    "one_long": [260] + [1] * 40,
    "last_chunk": [20] * 32 + [19],
}


def _csr(lens, seed):
    rng = np.random.default_rng(seed)
    row = np.concatenate([[0], np.cumsum(lens)]).astype(np.uint32)
    col = np.concatenate([np.sort(rng.choice(400, l, replace=False)) for l in lens])
    return row, col.astype(np.uint32), rng.standard_normal(int(row[-1]))


def _k1(row, arr, fill=0):
    lens = np.diff(row.astype(np.int64))
    perm, out = np.argsort(-lens, kind="stable"), []
    for c in range(0, len(perm), 32):
        rows = perm[c:c + 32]
        block = np.full((lens[rows[0]], 32), fill, arr.dtype)
        for lane, r in enumerate(rows):
            block[:lens[r], lane] = arr[row[r]:row[r + 1]]
        out.append(block.reshape(-1))
    return np.concatenate(out)


def _lens(name, l):
    return [l] * 70 if name == "uniform" else LENS[name]


CASES = [("uniform", l) for l in (1, 2, 3, 4, 5, 8, 9, 15, 16, 17, 127, 128, 129)] + \
    [(n, 0) for n in LENS if n != "uniform"]


@pytest.mark.parametrize("name,l", CASES)
@pytest.mark.parametrize("vtype", ["f64", "f32"])
@pytest.mark.parametrize("off", [0, 1, 3])
def test_slots(name, l, vtype, off):
    from gpu_spmv_b200 import engine as E

    row, col, val = _csr(_lens(name, l), 1)
    dt = torch.float64 if vtype == "f64" else torch.float32
    npt = np.float64 if vtype == "f64" else np.float32
    d_col = torch.from_numpy(np.concatenate([np.zeros(off, np.int32), col.view(np.int32)])).cuda()
    d_val = torch.from_numpy(np.concatenate([np.zeros(off), val])).to(dt).cuda()
    A = E.Matrix(row, d_col[off:], d_val[off:], ncols=400, fmt="K1", vtype=vtype, adjoint=True)
    lay = A.layout()
    assert np.array_equal(lay["val"], _k1(row, val.astype(npt)))
    assert np.array_equal(lay["col"], _k1(row, col))
    new = np.random.default_rng(2).standard_normal(len(val))
    src = torch.from_numpy(np.concatenate([np.zeros(off), new])).to(dt).cuda()[off:]
    A.set_values(src)
    assert np.array_equal(A.layout()["val"], _k1(row, new.astype(npt)))
    assert torch.equal(A.convert_values(A.convert_values(src, to="slots"), to="csr"), src)
    A.close()


@pytest.mark.parametrize("name,l", CASES)
@pytest.mark.parametrize("vtype", ["f32", "bf16"])
def test_blocked(name, l, vtype):
    from gpu_spmv_b200 import engine as E

    row, col, val = _csr(_lens(name, l), 3)
    x = torch.randn(400, device="cuda")
    ys = []
    for itype in ("u32", "u16"):
        A = E.Matrix(row, col, val, ncols=400, fmt="K1", vtype=vtype, itype=itype)
        ys.append(A.spmv(x, acc64=True))
        A.close()
    assert torch.equal(*ys)
