"""Operators beyond the persistent launch's range run pass by pass: the same bits with and without a
graph, and as with the launch disabled."""
import numpy as np
import pytest
import torch

import rqutils_b200 as rq

pytestmark = pytest.mark.gpu


def _full_space(n, masks):
    """All states of n qubits, masks + 1 pairs a row, real elements."""
    rng = np.random.default_rng(n + masks)
    x = np.concatenate([[0, 0, 0], 1 + rng.choice((1 << n) - 1, masks, replace=False)])
    x = x.astype(np.uint64)
    z = rng.integers(0, 1 << n, size=x.shape[0], dtype=np.uint64) & ~x
    ham = rq.PauliSumXZ.from_xz(x, z, rng.standard_normal(x.shape[0]), n, force_real=True,
                                padded=True)
    return rq.SQDOperator(ham, rq.Subspace.from_u64(np.arange(1 << n, dtype=np.uint64), n), (1, 2),
                          lookup='hash')


def _start(op, dt):
    return torch.randn(op.size, dtype=dt, generator=torch.Generator().manual_seed(3)).cuda()


@pytest.mark.parametrize('n, masks', [(19, 16), (20, 8), (21, 1)])
def test_long_operators_run_pass_by_pass(n, masks):
    op = _full_space(n, masks)
    x0 = _start(op, torch.float64)
    e0, v0, k0 = rq.ground_locg(op, x0, maxiter=6, use_graph=False)
    e1, v1, k1 = rq.ground_locg(op, x0, maxiter=6)
    assert e0 == e1 and k0 == k1 and torch.equal(v0, v1)


@pytest.mark.parametrize('n, masks', [(19, 16), (20, 8)])
def test_long_operators_mixed(n, masks, monkeypatch):
    op = _full_space(n, masks)
    x0 = _start(op, torch.float64)
    e1, v1, k1 = rq.ground_locg(op, x0, maxiter=6, mode='mixed')
    monkeypatch.setenv('SQD_LOCG_PERSISTENT', '0')
    e0, v0, k0 = rq.ground_locg(op, x0, maxiter=6, mode='mixed')
    assert e0 == e1 and k0 == k1 and torch.equal(v0, v1)
