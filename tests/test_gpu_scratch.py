"""The first multi-RHS call on a matrix allocates its scratch and waits for the stream, so that later
calls may come on any other stream that the caller orders behind it."""
import numpy as np
import pytest
import torch

from mats import csr_from_lengths

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("how", ["gs_spmm", "strided"])
def test_first_call_waits(how):
    from gpu_spmv_b200 import engine as E

    rng = np.random.default_rng(1)
    lens = rng.integers(0, 20, 500)
    lens[3] = 400  # a cut chunk: the scratch is used
    row, col, val = csr_from_lengths(lens, 500, rng)
    A, other = (E.Matrix(row, col, val, ncols=500, fmt="K1") for _ in range(2))
    X = torch.from_numpy(rng.standard_normal((500, 8))).cuda()
    X = X if how == "gs_spmm" else X[:, :3]
    want = other.spmm(X)  # loads the kernels, which waits by itself
    torch.cuda.synchronize()
    s, t = torch.cuda.Stream(), torch.cuda.Stream()
    queued = torch.cuda.Event()
    with torch.cuda.stream(s):
        torch.cuda._sleep(200_000_000)  # some 0.1 s
        queued.record()
        first = A.spmm(X)
        assert queued.query()
    t.wait_stream(s)
    with torch.cuda.stream(t):
        torch.cuda._sleep(200_000_000)
        queued.record()
        second = A.spmm(X)
        assert not queued.query()  # only the first call waits
    torch.cuda.synchronize()
    assert torch.equal(first, want) and torch.equal(second, want)
    A.close()
    other.close()
