"""SparseOperator stores the values of a call unless they are the stored ones: values that come to
lie at an earlier tensor's address, other views of one storage and values changed in place are
stored; the same ones again are not."""
import numpy as np
import pytest
import torch


class _Matrix:
    """Stands for engine.Matrix: remembers what was stored."""

    def __init__(self):
        self._stored = None
        self.calls = []

    def set_values(self, values, order="csr", stream=None):
        self.calls.append((values.clone(), order))


def _operator():
    from gpu_spmv_b200.autograd import SparseOperator

    op = SparseOperator.__new__(SparseOperator)
    op.mat = _Matrix()
    return op


def _ensure(op, v, order="csr"):
    op.ensure_values(v, order)
    last, o = op.mat.calls[-1]
    assert o == order and torch.equal(last, v)


def test_values_at_an_earlier_address():
    op = _operator()
    memory = np.zeros(1000)
    for step in range(4):
        memory[:] = step
        v = torch.from_numpy(memory)  # a new tensor, version 0, at the address of the last one
        _ensure(op, v)
        del v
    assert len(op.mat.calls) == 4


def test_views_of_one_storage():
    op = _operator()
    base = torch.arange(20.0)
    _ensure(op, base[:10])
    _ensure(op, base[::2])
    _ensure(op, base[10:])
    assert len(op.mat.calls) == 3


def test_changes_and_repeats():
    op = _operator()
    v = torch.zeros(5, requires_grad=True)
    for _ in range(3):
        _ensure(op, v.detach())
    assert len(op.mat.calls) == 1
    _ensure(op, v.detach(), "slots")
    with torch.no_grad():
        v += 1
    _ensure(op, v.detach(), "slots")
    assert len(op.mat.calls) == 3


@pytest.mark.gpu
@pytest.mark.parametrize("order", ["csr", "slots"])
def test_new_values_every_step(order):
    """Y and both gradients of steps that compute their values anew, against the fixed values'."""
    from gpu_spmv_b200.autograd import SparseOperator, spmm
    from mats import csr_from_lengths

    rng = np.random.default_rng(2)
    row, col, val = csr_from_lengths(rng.integers(0, 9, 300), 200, rng)
    op = SparseOperator(row, col, val, ncols=200)
    theta = torch.from_numpy(rng.standard_normal(len(col))).cuda()
    X = torch.from_numpy(rng.standard_normal((200, 4))).cuda()
    B = torch.from_numpy(rng.standard_normal((300, 4))).cuda()
    r = torch.from_numpy(np.repeat(np.arange(300), np.diff(row))).cuda()
    c = torch.from_numpy(col.astype(np.int64)).cuda()

    def step(i):
        t = theta.clone().requires_grad_()
        x = X.clone().requires_grad_()
        v = t * (i + 1.0)
        Y = spmm(v if order == "csr" else _slots(v), x, op, order=order)
        (Y * B).sum().backward()
        return Y.detach(), t.grad, x.grad

    def _slots(v):  # differentiable CSR -> slot order, through the operator's own index map
        idx = op.slot_values(torch.arange(1.0, len(col) + 1, dtype=torch.float64,
                                          device="cuda")).long()
        return torch.where(idx > 0, v[(idx - 1).clamp(min=0)], torch.zeros((), dtype=v.dtype,
                                                                         device=v.device))

    def product(out, i, j, v, D):  # out rows i gather v D[j]; and the same of the magnitudes
        zero = torch.zeros(out, 4, dtype=torch.float64, device="cuda")
        return (zero.index_add(0, i, v[:, None] * D[j]),
                zero.index_add(0, i, v.abs()[:, None] * D[j].abs()))

    def check(i):  # nothing outlives it: the next step's tensors take this one's places
        v = theta * (i + 1.0)
        g = (B[r] * X[c]) * (i + 1.0)
        # sums of at most 30 products
        for got, (want, mag) in zip(step(i), (product(300, r, c, v, X),
                                              (g.sum(1), g.abs().sum(1)),
                                              product(200, c, r, v, B))):
            assert torch.all((got - want).abs() <= 64 * 2.0 ** -53 * mag)

    for i in range(4):
        check(i)
    op.close()
