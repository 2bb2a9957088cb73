"""The FP64 reference iteration as one persistent launch (small operators with short rows) against
the same iteration launched pass by pass (use_graph=False), on one block, one cluster, and a grid
with barriers; real and complex, rows of one pair and of many."""
import numpy as np
import pytest
import torch

import rqutils_b200 as rq
from rqutils_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _op(n, weight, terms, dim, real, seed):
    rng = np.random.default_rng(seed)
    x, z, c = W.random_pauli_sum(n, terms, rng)
    if real:                               # an even number of Y per term
        odd = (np.bitwise_count(x & z) & 1).astype(bool)
        z[odd] ^= x[odd] & (~x[odd] + np.uint64(1))
    states = W.weight_subspace(n, weight, dim, rng)
    ham = rq.PauliSumXZ.from_xz(x, z, c, n, force_real=real, padded=True)
    return rq.SQDOperator(ham, rq.Subspace.from_u64(states, n), cache_strategy=(1, 2))


@pytest.mark.parametrize('n, weight, terms, dim', [
    (8, 4, 30, 3), (10, 5, 60, 251), (16, 8, 300, 2000), (16, 8, 300, 4096), (16, 8, 300, 4099),
    (20, 10, 1500, 12001), (30, 15, 900, 50001)])
@pytest.mark.parametrize('real', [True, False])
def test_persistent_equals_passes(n, weight, terms, dim, real):
    op = _op(n, weight, terms, dim, real, dim)
    assert op.nnz <= 36 * op.size
    dt = torch.float64 if real else torch.complex128
    gen = torch.Generator().manual_seed(5)
    x0 = torch.randn(op.size, dtype=dt, generator=gen).cuda()
    for maxiter in (1, 2, 3, 9, 10):
        e0, v0, k0 = rq.ground_locg(op, x0, maxiter=maxiter, use_graph=False)
        e1, v1, k1 = rq.ground_locg(op, x0, maxiter=maxiter)
        assert k0 == k1
        # the two differ in the order of the dots' sums: a few ulps an iteration, which the
        # iteration spreads over directions whose energies are close
        assert abs(e0 - e1) <= 1e-13 * max(1.0, abs(e0))
        assert (v0 - v1).abs().max() <= 1e-9
    e0, v0, k0 = rq.ground_locg(op, x0, use_graph=False)
    e1, v1, k1 = rq.ground_locg(op, x0)
    assert abs(e0 - e1) <= 1e-12 * max(1.0, abs(e0)) and abs(k0 - k1) <= 2
    assert abs(torch.linalg.vector_norm(v1).item() - 1.0) <= 1e-12
    res = torch.linalg.vector_norm(op.matvec(v1) - e1 * v1).item()
    ref = torch.linalg.vector_norm(op.matvec(v0) - e0 * v0).item()
    assert res <= 2.0 * ref + 1e-12


def test_start_vector_that_is_an_eigenvector():
    """A Z-only Hamiltonian: the start is exact and no iteration runs."""
    rng = np.random.default_rng(1)
    z = rng.integers(1, 1 << 10, size=40, dtype=np.uint64)
    c = rng.standard_normal(40)
    states = W.weight_subspace(10, 5, 200, rng)
    ham = rq.PauliSumXZ.from_xz(np.zeros_like(z), z, c, 10, force_real=True, padded=True)
    op = rq.SQDOperator(ham, rq.Subspace.from_u64(states, 10), cache_strategy=(1, 2))
    e, v, it = rq.ground_locg(op, op.vinit(), vspace=(op.size, torch.float64))
    assert it == 0 and e == op.diagonal(0).min().item()
