"""The converters' stable sort on the device: the K1 permutation (rows by decreasing length, ties
in row order) and the adjoint layout's order (elements by column, columns by decreasing count)
against numpy's stable argsort, at the edges of the sort's tiles (4096 elements) and of its passes
(at most 8 bits each).  Integers: equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _csr(lens, ncols, rng):
    row = np.zeros(len(lens) + 1, np.uint32)
    row[1:] = np.cumsum(lens)
    col = np.concatenate([np.sort(rng.choice(ncols, l, replace=False)) if l < 2000 else
                          np.arange(l) for l in lens] + [np.zeros(0, int)]).astype(np.uint32)
    return row, col, rng.standard_normal(len(col))


@pytest.mark.parametrize("n", [1, 32, 33, 4095, 4096, 4097, 12289])
@pytest.mark.parametrize("top", [0, 1, 255, 256, 65535, 65536])
def test_k1_permutation(n, top):
    from gpu_spmv_b200 import engine as E

    rng = np.random.default_rng(n + 7 * top)
    lens = np.minimum(rng.integers(0, 7, n), top)
    lens[n // 2] = top  # the longest row: `top` fixes the number of key bits
    row, col, val = _csr(lens, max(8, top), rng)
    A = E.Matrix(row, col, val, ncols=max(8, top), fmt="K1", keep_layout=True)
    assert np.array_equal(A.layout()["permi"][:n], np.argsort(-lens, kind="stable"))
    A.close()


@pytest.mark.parametrize("ncols", [1, 2, 256, 257, 70001])
@pytest.mark.parametrize("n", [1, 1365, 5000])
def test_adjoint_order(n, ncols):
    import torch

    from gpu_spmv_b200.autograd import SparseOperator

    rng = np.random.default_rng(n + ncols)
    row, col, val = _csr(np.minimum(rng.integers(0, 7, n), ncols), ncols, rng)
    nnz = len(col)
    op = SparseOperator(row, col, val, ncols=ncols, vtype="f64")
    ids = torch.arange(1, nnz + 1, dtype=torch.float64, device="cuda")
    got = op.slot_values(ids).cpu().numpy()
    count = np.bincount(col, minlength=ncols)
    csc, first = np.argsort(col, kind="stable"), np.concatenate([[0], np.cumsum(count)])
    want, perm = [], np.argsort(-count, kind="stable")
    for c in range(0, ncols, 32):
        chunk = perm[c:c + 32]
        block = np.zeros((count[chunk[0]], 32))
        for lane, j in enumerate(chunk):
            block[:count[j], lane] = csc[first[j]:first[j + 1]] + 1
        want.append(block.reshape(-1))
    assert np.array_equal(got, np.concatenate(want))
    op.close()
