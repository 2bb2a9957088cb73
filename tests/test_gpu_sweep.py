"""Connectivity by the (row, group) sweep on subspaces that are no product: row pointers, sources
and their order bit for bit against membership by sorted search, around the tile size, with one
and many group chunks, fill-in slots, and with more pairs than the sweep's buffer holds."""
import numpy as np
import pytest
import torch

import rqutils_b200 as rq
from rqutils_b200 import workloads as W
from oracle import symplectic as OS, sqd as OQ

pytestmark = pytest.mark.gpu


def _expected(ham, states, n, size):
    """(row pointers, sources): diagonal group first, then the groups on the high half only, on
    the low half only and on both, each in ascending mask order."""
    gx = ham.device_tables()[0].cpu().numpy().view(np.uint64)
    low = np.uint64((1 << (n // 2)) - 1)
    cls = np.where(gx == 0, 0, np.where((gx & low) == 0, 1, np.where((gx & ~low) == 0, 2, 3)))
    order = np.lexsort((gx, cls))
    nu = states.shape[0]
    rows, cols = [], []
    for j in order:
        want = states ^ gx[j]
        at = np.minimum(np.searchsorted(states, want), nu - 1)
        hit = np.nonzero(states[at] == want)[0]
        rows.append(hit)
        cols.append(at[hit])
    rows, cols = np.concatenate(rows), np.concatenate(cols)
    o = np.argsort(rows, kind='stable')
    rows, cols = rows[o], cols[o]
    counts = np.bincount(rows, minlength=size)
    if size > nu and gx[0] == 0:      # the last fill-in slot sources the first
        counts[size - 1] = 1
        cols = np.append(cols, nu)
    return np.concatenate([[0], np.cumsum(counts)]), cols


@pytest.mark.parametrize('n, weight, dim, terms, fill', [
    (16, 8, 2047, 300, 0), (16, 8, 2048, 40, 0), (17, 8, 2049, 900, 5), (40, 20, 5000, 3000, 0),
    (12, None, 1, 50, 0), (13, None, 700, 200, 3)])
def test_sweep_connectivity(n, weight, dim, terms, fill):
    rng = np.random.default_rng(dim + terms)
    x, z, c = W.random_pauli_sum(n, terms, rng)
    if weight is None:
        states = np.sort(rng.choice(1 << n, size=dim, replace=False)).astype(np.uint64)
    else:
        states = W.weight_subspace(n, weight, dim, rng)
    ham = rq.PauliSumXZ.from_xz(x, z, c, n, padded=True)
    space = rq.Subspace.from_u64(states, n, states_size=dim + fill)
    indptr, cols = _expected(ham, states, n, dim + fill)
    for lookup in ('hash', 'bsearch'):
        op = rq.SQDOperator(ham, space, cache_strategy=(1, 0), lookup=lookup)
        got = [t.cpu().numpy() for t in op.csr()[:2]]
        np.testing.assert_array_equal(got[0], indptr)
        np.testing.assert_array_equal(got[1], cols)


def test_more_pairs_than_the_buffer():
    """All 2^10 states, several hundred X masks: over 256 pairs per row, swept twice."""
    rng = np.random.default_rng(3)
    x, z, c = W.random_pauli_sum(10, 3000, rng, wmax=6)
    states = np.arange(1 << 10, dtype=np.uint64)
    ham = rq.PauliSumXZ.from_xz(x, z, c, 10, padded=True)
    space = rq.Subspace.from_u64(states, 10)
    indptr, cols = _expected(ham, states, 10, 1 << 10)
    assert indptr[-1] > (256 + 1) << 10
    op = rq.SQDOperator(ham, space, cache_strategy=(1, 2), lookup='hash')
    got = [t.cpu().numpy() for t in op.csr()[:2]]
    np.testing.assert_array_equal(got[0], indptr)
    np.testing.assert_array_equal(got[1], cols)


@pytest.mark.parametrize('dim', [511, 512, 1500])
def test_searching_matvec(dim):
    """The matvec that searches its sources (0, 0) around its tile size, against the oracle
    (apply_h_x_cached, sqd.py:694-709)."""
    rng = np.random.default_rng(dim)
    x, z, c = W.random_pauli_sum(16, 200, rng)
    states = W.weight_subspace(16, 8, dim, rng)
    ham = rq.PauliSumXZ.from_xz(x, z, c, 16, padded=True)
    op = rq.SQDOperator(ham, rq.Subspace.from_u64(states, 16), cache_strategy=(0, 0))
    oham = OS.from_paulisum((W.labels_from_xz(x, z, 16), list(c)), add_padding=True)
    sp = OQ.pack_states(OQ.u64_to_states(states, 16))
    xs = np.stack([OQ.get_xsource(xm, sp) for xm in oham.x])
    v = torch.randn(dim, dtype=torch.complex128, device='cuda')
    ref = OQ.apply_h_x_cached(v.cpu().numpy(), xs, oham.z, oham.c, sp)
    assert np.abs(op.matvec(v).cpu().numpy() - ref).max() <= 1e-13 * np.abs(ref).max()
