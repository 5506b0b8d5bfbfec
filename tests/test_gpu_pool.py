"""Device memory of matrices and conversion scratch: matrices made, used and destroyed by several
threads on their own streams give the products of a lone one, and gs_release_cached returns what a
destroyed matrix held."""
import threading

import numpy as np
import pytest
import torch

from mats import csr_from_lengths

pytestmark = pytest.mark.gpu


def _matrix(seed):
    rng = np.random.default_rng(seed)
    lens = rng.integers(0, 60, 3000 + 1000 * seed)
    lens[seed] = 900
    row, col, val = csr_from_lengths(lens, 5000, rng)
    return row, col, val, torch.from_numpy(rng.standard_normal(5000)).cuda()


def test_threads_and_streams():
    from gpu_spmv_b200 import engine as E

    cases = [_matrix(i) for i in range(4)]
    fmts = [dict(fmt="K1"), dict(fmt="CSR"), dict(fmt="AXT", mode="UNC", tileH=4), dict(fmt="AXC")]

    def product(i, fmt):
        row, col, val, x = cases[i]
        A = E.Matrix(row, col, val, ncols=5000, **fmt)
        y = A.spmv(x)
        A.close()
        return y

    want = [[product(i, f).clone() for f in fmts] for i in range(4)]
    torch.cuda.synchronize()
    bad = []

    def work(i):
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            for _ in range(15):
                for f, w in zip(fmts, want[i]):
                    y = product(i, f)
                    s.synchronize()
                    if not torch.equal(y, w):
                        bad.append((i, f))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


def test_release_cached():
    from gpu_spmv_b200 import _lib as L
    from gpu_spmv_b200 import engine as E

    rng = np.random.default_rng(5)
    row, col, val = csr_from_lengths(np.full(100000, 50), 200000, rng)
    A = E.Matrix(row, col, val, ncols=200000, fmt="K1")
    held = A.info.nslots * 12
    A.close()
    before = torch.cuda.mem_get_info()[0]
    L.check(L.lib().gs_release_cached(), "gs_release_cached")
    assert torch.cuda.mem_get_info()[0] - before >= held


def test_release_cached_python():
    """A Python program gives the memory of closed matrices back without the C library."""
    from gpu_spmv_b200 import engine as E

    rng = np.random.default_rng(6)
    row, col, val = csr_from_lengths(np.full(100000, 50), 200000, rng)
    A = E.Matrix(row, col, val, ncols=200000, fmt="K1")
    held = A.info.nslots * 12
    A.close()
    before = torch.cuda.mem_get_info()[0]
    E.release_cached()
    assert torch.cuda.mem_get_info()[0] - before >= held
    E.release_cached("cuda:0")
