"""Elements of product subspaces too small or too narrow for the halves' kernels: the same numbers
in the pair list and in the slabs, and no slower than without the lists."""
import numpy as np
import pytest
import torch

import rqutils_b200 as rq
from rqutils_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _operators(na, nb, real):
    wl = W.jw_workload('routes', 12, 4, na, nb, 4)
    ham = rq.PauliSumXZ.from_xz(wl.x, wl.z, wl.coeffs, 24, force_real=True, padded=True)
    space = rq.Subspace.from_u64(wl.states, 24)
    return ham, wl.coeffs, [rq.SQDOperator(ham, space, (1, 2), lookup=k)
                            for k in ('product', 'hash')]


@pytest.mark.parametrize('na, nb', [(495, 1), (1, 495), (64, 60), (240, 239), (495, 120)])
def test_elements_and_slabs_after_a_refresh(na, nb):
    ham, c, ops = _operators(na, nb, True)
    for op in ops:
        op.set_layout(0, 'product')
        op.set_layout(1, 'product')
    ham.set_coeffs(torch.as_tensor(0.7 * c - 0.2))
    for op in ops:
        op.refresh()
    for a, b in zip(ops[0].csr(), ops[1].csr()):
        assert torch.equal(a, b)
    for dt in (torch.float64, torch.complex64):
        prec = 0 if dt == torch.float64 else 1
        v = torch.randn(ops[0].size, dtype=dt, device='cuda')
        assert torch.equal(ops[0].matvec(v), ops[1].matvec(v))
        ref = ops[0].matvec(v)
        ops[0].set_layout(prec, 'csr')
        eps = torch.finfo(dt).eps
        # at most 500 products a row, in two orders
        assert (ops[0].matvec(v) - ref).abs().max() <= 500 * eps * ref.abs().max()


@pytest.mark.parametrize('na, nb', [(495, 1), (1, 495)])
def test_one_string_in_a_half_is_not_slower(na, nb):
    """Seven times the time of the row by row kernels, when a warp summed a string's list."""
    _, _, ops = _operators(na, nb, True)
    times = []
    for op in ops:
        best = float('inf')
        for _ in range(5):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            op.refresh()
            a.record()
            for _ in range(20):
                op.refresh()
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b))
        times.append(best)
    assert times[0] <= 2.5 * times[1]
