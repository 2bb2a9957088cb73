"""Per-term sums at the ends of their range, against sums in PyTorch."""
import numpy as np
import pytest
import torch

import rqutils_b200 as rq

pytestmark = pytest.mark.gpu


def test_diagonal_group_of_millions_of_terms():
    n, terms = 23, 65535 * 64 + 70
    rng = np.random.default_rng(2)
    z = np.arange(1, terms + 1, dtype=np.uint64)
    ham = rq.PauliSumXZ.from_xz(np.zeros_like(z), z, np.ones(terms), n, force_real=True,
                                padded=True)
    states = np.sort(rng.choice(1 << n, size=40, replace=False)).astype(np.uint64)
    op = rq.SQDOperator(ham, rq.Subspace.from_u64(states, n), cache_strategy=(1, 0))
    u, v = (torch.randn(op.size, dtype=torch.float64, device='cuda') for _ in range(2))
    got = op.grad_terms(u, v)[ham.raw_to_term()]
    zt = torch.arange(1, terms + 1, device='cuda')
    want = torch.zeros(terms, dtype=torch.float64, device='cuda')
    for s, w in zip(states.tolist(), (u * v).tolist()):
        b = zt & s
        for k in (16, 8, 4, 2, 1):
            b = b ^ (b >> k)
        want += w * (1 - 2 * (b & 1)).double()
    # 40 products a term
    assert (got - want).abs().max() <= 80 * 2.0 ** -52 * (u * v).abs().sum()
