"""Where the partner lists of a product subspace are the slower way, the composing matvec is the one
that an explicit lookup gives: the same sums in the same order, so the same bits."""
import numpy as np
import pytest
import torch

import rqutils_b200 as rq
from rqutils_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _heavy(n, terms, real, rng):
    """Strings with a letter on every other qubit: nearly every group acts on both halves, and a
    few hundred of them give tens of thousands of combinations of their halves' parts."""
    x = rng.integers(1, 1 << n, size=terms, dtype=np.uint64)
    z = rng.integers(0, 1 << n, size=terms, dtype=np.uint64)
    if real:
        z &= ~x
    return x, z, rng.standard_normal(terms)


def _case(name):
    rng = np.random.default_rng(21)
    if name.startswith('jw'):
        na, nb = {'jw-tile': (32, 32), 'jw-100': (56, 50), 'jw-3': (3, 56), 'jw-1': (1, 56)}[name]
        wl = W.jw_workload(name, 8, 3, na, nb, 3)
        return wl.x, wl.z, wl.coeffs, wl.states, 16
    if name == 'ising':
        n = 14
        bond = np.array([3 << q for q in range(n - 1)], dtype=np.uint64)
        x = np.concatenate([np.zeros_like(bond), np.uint64(1) << np.arange(n, dtype=np.uint64)])
        z = np.concatenate([bond, np.zeros(n, dtype=np.uint64)])
        return x, z, rng.standard_normal(x.shape[0]), np.arange(1 << n, dtype=np.uint64), n
    if name == 'sparse':              # many rows, a combination in a hundred has a group
        n = 18
        x, z, c = _heavy(n, 40, True, rng)
    else:
        n = 14
        x, z, c = _heavy(n, 300, True, rng)
    return x, z, c, np.arange(1 << n, dtype=np.uint64), n


CASES = [(name, (1, 0)) for name in ('jw-tile', 'jw-100', 'jw-3', 'jw-1', 'ising', 'sparse',
                                     'heavy')] + [('sparse', (0, 0)), ('heavy', (0, 0))]


@pytest.mark.parametrize('name, cache', CASES)
def test_lists_are_not_taken(name, cache):
    x, z, c, states, n = _case(name)
    ham = rq.PauliSumXZ.from_xz(x, z, c, n, force_real=True, padded=True)
    space = rq.Subspace.from_u64(states, n)
    ops = [rq.SQDOperator(ham, space, cache_strategy=cache, lookup=k) for k in ('auto', 'hash')]
    assert ops[0].nnz == ops[1].nnz
    for dt in (torch.complex128, torch.float64, torch.complex64, torch.float32):
        gen = torch.Generator().manual_seed(2)
        v = torch.randn(states.shape[0], generator=gen, dtype=dt).cuda()
        assert torch.equal(ops[0].matvec(v), ops[1].matvec(v)), dt
