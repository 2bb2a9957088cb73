"""Partner lists of more strings than the grid has blocks: the connectivity equals the sweep's."""
import numpy as np
import pytest
import torch

import rqutils_b200 as rq

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('high', [True, False])
def test_strings_beyond_the_grid(high):
    bits, count = 22, (1 << 20) + 77
    rng = np.random.default_rng(3)
    states = np.sort(rng.choice(1 << bits, size=count, replace=False)).astype(np.uint64)
    x = np.array([0, 1, 6, 40, 0x300, 0x2001, 0x100000, 0x3], dtype=np.uint64)
    if high:
        states, x = states << np.uint64(bits), x << np.uint64(bits)
    ham = rq.PauliSumXZ.from_xz(x, np.zeros_like(x), rng.standard_normal(x.shape[0]), 2 * bits,
                                force_real=True, padded=True)
    space = rq.Subspace.from_u64(states, 2 * bits)
    a = rq.SQDOperator(ham, space, cache_strategy=(1, 2), lookup='product').csr()
    b = rq.SQDOperator(ham, space, cache_strategy=(1, 2), lookup='hash').csr()
    for u, w in zip(a, b):
        assert torch.equal(u, w)
