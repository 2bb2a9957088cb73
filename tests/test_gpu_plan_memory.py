"""Strategy (0, 0) keeps nothing that grows like a pair list: one string in a half."""
import numpy as np
import pytest
import torch

import rqutils_b200 as rq
from rqutils_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('high', [True, False])
def test_uncached_operator_of_a_lopsided_product(high):
    bits = 21
    x = np.array([0, 3, 5, 9, 17, 33, 65, 129, 257, 513, 1025, 2049, 6, 12, 24, 48, 96],
                 dtype=np.uint64)
    states = np.arange(1 << bits, dtype=np.uint64)
    if high:
        x, states = x << np.uint64(bits), states << np.uint64(bits)
    rng = np.random.default_rng(1)
    ham = rq.PauliSumXZ.from_xz(x, np.zeros_like(x), rng.standard_normal(x.shape[0]), 2 * bits,
                                force_real=True, padded=True)
    space = rq.Subspace.from_u64(states, 2 * bits)
    torch.cuda.synchronize()
    used = _lib.memory_stats()[1]
    op = rq.SQDOperator(ham, space, cache_strategy=(0, 0))
    torch.cuda.synchronize()
    assert _lib.memory_stats()[1] - used <= 64 << 20      # 33.5 M entries would be 268 MB
    v = torch.randn(op.size, dtype=torch.float64, device='cuda')
    ref = rq.SQDOperator(ham, space, cache_strategy=(0, 0), lookup='hash').matvec(v)
    assert torch.equal(op.matvec(v), ref)
