"""Two-half pairs of the product layout in panels: every size class of the kernel (panels per
warp, several blocks per high string, rows too long for shared memory), absent combinations and
non-finite amplitudes, against the pair-list layout of the same operator."""
import numpy as np
import pytest
import torch

import rqutils_b200 as rq

pytestmark = pytest.mark.gpu


def _operator(nh, nl, half, missing, cplx, seed):
    """nh x nl random strings of `half` bits each; two-half groups over 5 x 9 parts, `missing` of
    them dropped; single-half groups and a diagonal beside them."""
    rng = np.random.default_rng(seed)
    hi = np.sort(rng.choice(1 << half, size=nh, replace=False)).astype(np.uint64)
    lo = np.sort(rng.choice(1 << half, size=nl, replace=False)).astype(np.uint64)
    states = ((hi[:, None] << np.uint64(half)) | lo[None, :]).reshape(-1)
    # high parts that connect the drawn strings, low parts of one or two bits
    xa = np.unique(np.concatenate([hi[:1] ^ hi[1:6], hi[2:3] ^ hi[:2]]))
    xa = xa[xa != 0][:5]
    xb = np.array([1, 2, 3, 4, 5, 6, 8, 9, 12], dtype=np.uint64)
    pairs = [(a, b) for a in xa for b in xb]
    drop = set(rng.choice(len(pairs), size=int(missing * len(pairs)), replace=False).tolist())
    x = [(int(a) << half) | int(b) for i, (a, b) in enumerate(pairs) if i not in drop]
    x = x + [int(a) << half for a in xa] + [int(b) for b in xb] + [0]
    x = np.repeat(np.array(x, dtype=np.uint64), 3)
    z = rng.integers(0, 1 << (2 * half), size=x.shape[0], dtype=np.uint64)
    c = rng.standard_normal(x.shape[0])
    if not cplx:                      # an even number of Y per term: real elements
        odd = (np.bitwise_count(x & z) & 1).astype(bool)
        z[odd] ^= x[odd] & (~x[odd] + np.uint64(1))
    n = 2 * half
    ham = rq.PauliSumXZ.from_xz(x, z, c, n, force_real=not cplx, padded=True)
    op = rq.SQDOperator(ham, rq.Subspace.from_u64(states, n), cache_strategy=(1, 2))
    assert op.value_complex == cplx
    return ham, op, c


SIZES = [(33, 1, 8), (34, 31, 8), (40, 64, 8), (20, 1025, 11), (16, 2500, 13), (12, 4000, 13),
         (9, 4300, 13), (7, 6500, 14)]


@pytest.mark.parametrize('nh, nl, half', SIZES)
@pytest.mark.parametrize('cplx', [False, True])
def test_panels_match_the_pair_list(nh, nl, half, cplx):
    for missing in (0.0, 0.2):
        ham, op, c = _operator(nh, nl, half, missing, cplx, nl)
        types = [torch.complex128, torch.complex64]
        if not cplx:
            types += [torch.float64, torch.float32]
        for coeffs in (c, 0.6 * c + 0.1):
            if coeffs is not c:
                ham.set_coeffs(torch.as_tensor(coeffs))
                op.refresh()
            for dt in types:
                prec = 0 if dt in (torch.complex128, torch.float64) else 1
                gen = torch.Generator().manual_seed(nh)
                v = torch.randn(op.size, dtype=dt, generator=gen).cuda()
                op.set_layout(prec, 'csr')
                ref = op.matvec(v)
                op.set_layout(prec, 'product')
                got = op.matvec(v)
                # at most 60 products a row: both sums within 60 ulps of the largest row's scale
                eps = torch.finfo(dt).eps * 60 * 4
                assert (got - ref).abs().max() <= eps * ref.abs().max(), (dt, missing)
                op.set_layout(prec, 'product-csr')
                assert (op.matvec(v) - ref).abs().max() <= eps * ref.abs().max(), (dt, missing)


@pytest.mark.parametrize('dt', [torch.float64, torch.complex64])
def test_absent_combinations_read_no_amplitude(dt):
    """An infinite amplitude reaches the rows connected to it and no others."""
    ham, op, c = _operator(24, 70, 8, 0.3, False, 5)
    prec = 0 if dt == torch.float64 else 1
    v = torch.ones(op.size, dtype=dt, device='cuda')
    for j in (0, 35, op.size - 1):
        v[j] = float('inf')
    op.set_layout(prec, 'csr')
    ref = torch.isfinite(op.matvec(v).abs())
    op.set_layout(prec, 'product')
    assert torch.equal(torch.isfinite(op.matvec(v).abs()), ref)
