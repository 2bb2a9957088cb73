"""Matrix elements of the stored pairs (cached, and re-composed after a coefficient update): every
element equals the group's terms summed in the reference's order (get_diagonal,
sqd.py:603-628), bit for bit, on general and on product subspaces."""
import numpy as np
import pytest
import torch

import rqutils_b200 as rq
from rqutils_b200 import workloads as W
from oracle import symplectic as OS

pytestmark = pytest.mark.gpu


def _cases():
    # JW, 8 orbitals: two-body groups, one-body groups of up to 30 terms, a 137-term diagonal
    jw = W.jw_workload('jw', 8, 3, 37, 33, 5)
    yield 'product', jw.x, jw.z, jw.coeffs, jw.states, 16, True
    rng = np.random.default_rng(2)
    some = np.sort(rng.choice(jw.states, size=701, replace=False))
    yield 'sampled', jw.x, jw.z, jw.coeffs, some, 16, True
    # few X masks with many Z masks each: groups of 23..26 and more terms, complex elements
    masks = np.array([0, 3, 5, 6, 0x300, 0x900, 0x303, 0x905], dtype=np.uint64)
    x = np.repeat(masks, [40, 23, 24, 25, 26, 70, 24, 25])
    z = np.concatenate([rng.choice(1 << 12, size=k, replace=False).astype(np.uint64)
                        for k in (40, 23, 24, 25, 26, 70, 24, 25)])
    c = rng.standard_normal(x.shape[0])
    yield 'long-product', x, z, c, W.product_subspace(6, 3, 17, 19, rng), 12, False
    yield 'long-general', x, z, c, np.sort(rng.choice(1 << 12, size=997, replace=False)
                                           ).astype(np.uint64), 12, False


CASES = {c[0]: c[1:] for c in _cases()}


def _expected(ham, states, indptr, indices):
    """Elements in CSR order: NumPy, one group at a time, terms added in stored order."""
    gx, gs, tz, tc, _ = (t.cpu().numpy() for t in ham.device_tables())
    gx, tz = gx.view(np.uint64), tz.view(np.uint64)
    group = {int(v): j for j, v in enumerate(gx)}
    rows = np.repeat(np.arange(indptr.shape[0] - 1), np.diff(indptr))
    out = np.zeros(indices.shape[0], dtype=np.complex128)
    j = np.array([group[int(v)] for v in states[rows] ^ states[indices]])
    for g in np.unique(j):
        at = np.nonzero(j == g)[0]
        s = states[rows[at]]
        acc = np.zeros(at.shape[0], dtype=np.complex128)
        for t in range(gs[g], gs[g + 1]):
            sign = 1.0 - 2.0 * (np.bitwise_count(s & tz[t]) & 1)
            acc = acc + tc[t] * sign
        out[at] = acc
    return out


@pytest.mark.parametrize('name', list(CASES))
def test_elements_equal_ordered_sums(name):
    x, z, c, states, n, real = CASES[name]
    ham = rq.PauliSumXZ.from_xz(x, z, c, n, force_real=real, padded=True)
    op = rq.SQDOperator(ham, rq.Subspace.from_u64(states, n), cache_strategy=(1, 2))
    v = torch.randn(op.size, dtype=torch.complex128, device='cuda')
    for coeffs in (c, c * 0.37 + 0.01):
        if coeffs is not c:
            ham.set_coeffs(torch.as_tensor(coeffs))
            stale = op.matvec(v)            # elements stay until the refresh
            assert torch.equal(stale, hv)
            op.refresh()
        hv = op.matvec(v)
        indptr, indices, data = (t.cpu().numpy() for t in op.csr())
        want = _expected(ham, states, indptr, indices)
        np.testing.assert_array_equal(data, want)
        # the cached elements are the exported ones: each row summed with its own vector entries
        # against a different association, so to rounding
        rows = np.repeat(np.arange(op.size), np.diff(indptr))
        ref = np.zeros(op.size, dtype=np.complex128)
        np.add.at(ref, rows, want * v.cpu().numpy()[indices])
        scale = np.zeros(op.size)
        np.add.at(scale, rows, np.abs(want) * np.abs(v.cpu().numpy()[indices]))
        longest = int(np.diff(indptr).max())
        bound = 4 * (longest + 4) * np.finfo(float).eps * scale.max()
        assert np.abs(hv.cpu().numpy() - ref).max() <= bound
        assert op.vinit() == int(np.argmin(want.real[indptr[:-1]]))


@pytest.mark.parametrize('name', ['product', 'long-product'])
def test_slabs_follow_a_refresh_and_not_the_coefficients(name):
    """Slabs selected after set_coeffs without a refresh hold the operator's own elements (as its
    pair list does); the refresh updates both."""
    x, z, c, states, n, real = CASES[name]
    ham = rq.PauliSumXZ.from_xz(x, z, c, n, force_real=real, padded=True)
    op = rq.SQDOperator(ham, rq.Subspace.from_u64(states, n), cache_strategy=(1, 2))
    v = torch.randn(op.size, dtype=torch.complex128, device='cuda')
    tol = {0: 1e-13, 1: 2e-6}
    before = op.matvec(v)
    ham.set_coeffs(torch.as_tensor(2.0 * c))
    for prec, dt in ((0, torch.complex128), (1, torch.complex64)):
        op.set_layout(prec, 'product')
        got = op.matvec(v.to(dt)).to(torch.complex128)
        assert (got - before).abs().max() <= tol[prec] * before.abs().max()
    op.refresh()
    for prec, dt in ((0, torch.complex128), (1, torch.complex64)):
        got = op.matvec(v.to(dt)).to(torch.complex128)
        assert (got - 2.0 * before).abs().max() <= tol[prec] * 2.0 * before.abs().max()
