"""Sweep-built operators whose rows are mostly fill-in slots (many repeats of few states): the
connectivity, and memory that follows the states and not the slots."""
import numpy as np
import pytest
import torch

import rqutils_b200 as rq
from rqutils_b200 import _lib
from rqutils_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('diagonal', [True, False])
def test_many_fill_in_slots(diagonal):
    n, dim, size = 30, 1500, 2_000_000
    rng = np.random.default_rng(8)
    # every even mask on 14 qubits: 8,191 groups that can connect, 128 chunks of 64
    x = np.arange(1 << 14, dtype=np.uint64)
    x = x[np.bitwise_count(x) % 2 == 0][0 if diagonal else 1:]
    z = rng.integers(0, 1 << n, size=x.shape[0], dtype=np.uint64)
    states = W.weight_subspace(14, 7, dim, rng)
    ham = rq.PauliSumXZ.from_xz(x, z, rng.standard_normal(x.shape[0]), n, padded=True)
    space = rq.Subspace.from_u64(states, n, states_size=size)
    few = rq.SQDOperator(ham, rq.Subspace.from_u64(states, n), (1, 2), 'hash').csr()
    torch.cuda.synchronize()
    _, used, _ = _lib.memory_stats(reset_high=True)
    op = rq.SQDOperator(ham, space, cache_strategy=(1, 2))
    torch.cuda.synchronize()
    # row pointers and their scan take 16 bytes a slot; counts per slot and chunk were 1 KB
    assert _lib.memory_stats()[2] - used < 64 * size + (64 << 20)
    indptr, cols, data = op.csr()
    nnz = few[1].shape[0]
    assert op.nnz == nnz + int(diagonal)
    assert torch.equal(indptr[:dim + 1], few[0])
    assert bool((indptr[dim + 1:size] == nnz).all()) and indptr[size].item() == op.nnz
    assert torch.equal(cols[:nnz], few[1]) and torch.equal(data[:nnz], few[2])
    if diagonal:
        assert cols[nnz].item() == dim
        assert data[nnz] == op.diagonal(0, torch.complex128)[size - 1]
