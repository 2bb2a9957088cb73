"""Matvec of a product subspace without stored elements (cache strategies (0, *), (1, 0), (1, 1)):
pairs from the halves' partner lists, elements composed; against the CPU oracle
(apply_h_x_cached, sqd.py:694-709) and the searching matvec."""
import numpy as np
import pytest
import torch

import rqutils_b200 as rq
from rqutils_b200 import workloads as W
from oracle import symplectic as OS, sqd as OQ

pytestmark = pytest.mark.gpu
RTOL = {torch.complex128: 1e-13, torch.float64: 1e-13, torch.complex64: 2e-6,
        torch.float32: 2e-6}


def _sub(n, nh, nl, rng):
    hi = np.sort(rng.choice(1 << (n - n // 2), size=nh, replace=False)).astype(np.uint64)
    lo = np.sort(rng.choice(1 << (n // 2), size=nl, replace=False)).astype(np.uint64)
    return ((hi[:, None] << np.uint64(n // 2)) | lo[None, :]).reshape(-1)


def _case(name):
    rng = np.random.default_rng(17)
    if name.startswith('jw'):
        na, nb = {'jw-tile': (32, 32), 'jw-ragged': (33, 45), 'jw-small': (31, 3)}[name]
        wl = W.jw_workload(name, 8, 3, na, nb, 3)
        return wl.x, wl.z, wl.coeffs, wl.states, 16, True
    # general Pauli sums: no conserved weight, complex elements, odd qubit number
    nh, nl, nodiag = {'random': (40, 50, False), 'one-high': (1, 64, False),
                      'one-low': (65, 1, False), 'no-diagonal': (20, 33, True)}[name]
    x, z, c = W.random_pauli_sum(13, 400, rng, wmax=4)
    if nodiag:
        x, z, c = x[x != 0], z[x != 0], c[x != 0]
    return x, z, c, _sub(13, nh, nl, rng), 13, False


@pytest.mark.parametrize('name', ['jw-tile', 'jw-ragged', 'jw-small', 'random', 'one-high',
                                  'one-low', 'no-diagonal'])
def test_composed_matvec_on_product_subspaces(name):
    x, z, c, states, n, real = _case(name)
    ham = rq.PauliSumXZ.from_xz(x, z, c, n, force_real=real, padded=True)
    space = rq.Subspace.from_u64(states, n)
    oham = OS.from_paulisum((W.labels_from_xz(x, z, n), list(c)), force_real=real,
                            add_padding=True)
    sp = OQ.pack_states(OQ.u64_to_states(states, n))
    xs = np.stack([OQ.get_xsource(xm, sp) for xm in oham.x])
    types = [torch.complex128, torch.complex64]
    if not ham.is_complex:
        types += [torch.float64, torch.float32]
    for dt in types:
        gen = torch.Generator().manual_seed(4)
        v = torch.randn(states.shape[0], generator=gen, dtype=dt).cuda()
        ref = OQ.apply_h_x_cached(v.cpu().numpy().astype(np.complex128), xs, oham.z, oham.c, sp)
        scale = np.abs(ref).max()
        for cache in ((0, 0), (0, 2), (1, 0), (1, 1)):
            for lookup in ('auto', 'hash'):
                op = rq.SQDOperator(ham, space, cache_strategy=cache, lookup=lookup)
                got = op.matvec(v).cpu().numpy()
                assert np.abs(got - ref).max() <= RTOL[dt] * scale, (dt, cache, lookup)


@pytest.mark.parametrize('nh, nl', [(1, 70001), (33000, 3)])
def test_many_strings_in_one_half(nh, nl):
    """More strings than get eight warps each: the connectivity equals the sweep's."""
    rng = np.random.default_rng(nh)
    hi = np.sort(rng.choice(1 << 17, size=nh, replace=False)).astype(np.uint64)
    lo = np.sort(rng.choice(1 << 17, size=nl, replace=False)).astype(np.uint64)
    states = ((hi[:, None] << np.uint64(17)) | lo[None, :]).reshape(-1)
    x, z, c = W.random_pauli_sum(34, 150, rng, wmax=3)
    ham = rq.PauliSumXZ.from_xz(x, z, c, 34, padded=True)
    space = rq.Subspace.from_u64(states, 34)
    a = rq.SQDOperator(ham, space, cache_strategy=(1, 2), lookup='product').csr()
    b = rq.SQDOperator(ham, space, cache_strategy=(1, 2), lookup='hash').csr()
    for u, w in zip(a, b):
        assert torch.equal(u, w)
