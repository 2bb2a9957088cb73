"""Per-term sums at the ends of their range, against sums in PyTorch."""
import numpy as np
import pytest
import torch

import rqutils_b200 as rq
from rqutils_b200 import _lib

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


@pytest.mark.parametrize('dt', [torch.float64, torch.complex128])
def test_groups_of_many_pairs(dt):
    """Few masks on a nearly full space: every group's 60,000 pairs have several owners; groups of
    one term, of more than a warp's eight and of more than a block's 64."""
    n, nh, nl = 16, 250, 251
    rng = np.random.default_rng(4)
    hi = np.sort(rng.choice(256, size=nh, replace=False)).astype(np.uint64)
    lo = np.sort(rng.choice(256, size=nl, replace=False)).astype(np.uint64)
    states = ((hi[:, None] << np.uint64(8)) | lo[None, :]).reshape(-1)
    x = np.repeat(np.array([0, 0x300, 0x500, 0x5, 0x9, 0x303, 0x509], dtype=np.uint64),
                  [3, 1, 70, 9, 130, 9, 1])
    z = rng.integers(0, 1 << n, size=x.shape[0], dtype=np.uint64)
    if dt == torch.float64:                 # an even number of Y per term
        odd = (np.bitwise_count(x & z) & 1).astype(bool)
        z[odd] ^= x[odd] & (~x[odd] + np.uint64(1))
    ham = rq.PauliSumXZ.from_xz(x, z, rng.standard_normal(x.shape[0]), n,
                                force_real=dt == torch.float64, padded=True)
    op = rq.SQDOperator(ham, rq.Subspace.from_u64(states, n), cache_strategy=(1, 2))
    gen = torch.Generator().manual_seed(1)
    u, v = (torch.randn(op.size, dtype=dt, generator=gen).cuda() for _ in range(2))
    got = op.grad_terms(u, v)[ham.raw_to_term()].cpu()
    s = torch.as_tensor(states.astype(np.int64))
    at = torch.full((1 << n,), -1, dtype=torch.int64)
    at[s] = torch.arange(op.size)
    u, v = u.cpu().to(torch.complex128), v.cpu().to(torch.complex128)
    for k in range(x.shape[0]):
        xk, zk = int(x[k]), int(z[k])
        src = at[s ^ xk]
        w = torch.where(src >= 0, u.conj() * v[src.clamp(min=0)], 0.0)
        b = s & zk
        for q in (8, 4, 2, 1):
            b = b ^ (b >> q)
        want = ((-1j) ** (bin(xk & zk).count('1') & 3) * (1 - 2 * (b & 1)).double() * w).real.sum()
        # 60,000 products, each rounded by a few ulps, in chains of at most 4096
        assert abs(got[k] - want) <= 4 * 2.0 ** -52 * op.size ** 0.5 * w.abs().sum(), k


@pytest.mark.slow
def test_more_list_entries_than_the_sort_takes():
    """One high string and 2^26 low ones with 32 masks: 2^31 list entries, summed pair by pair."""
    bits = 26
    x = np.concatenate([1 << np.arange(bits, dtype=np.uint64), np.array([3, 5, 9, 17, 33, 65],
                                                                        dtype=np.uint64)])
    z = np.zeros_like(x)
    z[::2] = np.uint64(1 << 12)
    z &= ~x
    ham = rq.PauliSumXZ.from_xz(x, z, np.ones(x.shape[0]), 2 * bits, force_real=True, padded=True)
    states = torch.arange(1 << bits, dtype=torch.int64, device='cuda')
    op = rq.SQDOperator(ham, rq.Subspace.from_u64(states, 2 * bits), cache_strategy=(1, 0))
    assert op.nnz == 1 << 31
    gen = torch.Generator(device='cuda').manual_seed(1)
    u, v = (torch.randn(op.size, dtype=torch.float64, generator=gen, device='cuda')
            for _ in range(2))
    got = op.grad_terms(u, v)[ham.raw_to_term()]
    for k in range(x.shape[0]):
        w = u * v[states ^ int(x[k])]
        want = (w * (1 - 2 * ((states & int(z[k])) != 0).double())).sum()
        # 2^26 products added one by one: a random walk of rounding errors of the partial sums
        assert (got[k] - want).abs() <= 2.0 ** -52 * op.size ** 0.5 * w.abs().sum(), k
    del op
    _lib.trim_memory()
