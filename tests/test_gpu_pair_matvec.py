"""The FP64 iteration applies its operator to y and p in one pass over the elements: same energies,
iteration counts and vectors, bit for bit, as with one matvec at a time (the operator passed as a
plain callable), and the oracle's iteration agrees."""
import numpy as np
import pytest
import torch

import rqutils_b200 as rq
from rqutils_b200 import workloads as W
from oracle import ground_locg as OL

pytestmark = pytest.mark.gpu


def _op(name):
    rng = np.random.default_rng(9)
    if name == 'complex':                       # odd-Y terms on a product of random halves
        x, z, c = W.random_pauli_sum(16, 700, rng, wmax=4)
        states, real, n = W.product_subspace(8, 4, 70, 65, rng), False, 16
    elif name == 'large':                       # above the pair list's threshold
        wl = W.jw_workload(name, 16, 4, 131, 129, 2)
        x, z, c, states, real, n = wl.x, wl.z, wl.coeffs, wl.states, True, 32
    else:                                       # ragged panels, short and long tails
        na, nb = {'jw': (20, 24), 'odd': (55, 37), 'one': (33, 1)}[name]
        wl = W.jw_workload(name, 8, 3, na, nb, 2)
        x, z, c, states, real, n = wl.x, wl.z, wl.coeffs, wl.states, True, 16
    ham = rq.PauliSumXZ.from_xz(x, z, c, n, force_real=real, padded=True)
    return rq.SQDOperator(ham, rq.Subspace.from_u64(states, n), cache_strategy=(1, 2))


@pytest.mark.parametrize('name', ['jw', 'odd', 'one', 'complex', 'large'])
@pytest.mark.parametrize('dt', [torch.float64, torch.complex128])
def test_pair_equals_single_matvecs(name, dt, monkeypatch):
    # pass by pass: the persistent launch of short-row operators sums its dots in another order
    monkeypatch.setenv('SQD_LOCG_PERSISTENT', '0')
    op = _op(name)
    if op.value_complex and not dt.is_complex:
        pytest.skip('complex elements need complex vectors')
    gen = torch.Generator().manual_seed(1)
    x0 = torch.randn(op.size, dtype=dt, generator=gen).cuda()
    for layout in ('csr', 'product', 'product-csr'):
        op.set_layout(0, layout)
        want = rq.ground_locg(op.matvec, x0, maxiter=15)
        for graph in (True, False):
            got = rq.ground_locg(op, x0, maxiter=15, use_graph=graph)
            assert got[0] == want[0] and got[2] == want[2], (layout, graph)
            assert torch.equal(got[1], want[1]), (layout, graph)


def test_constrained_iteration_and_oracle():
    """With an orthogonality constraint (A x recomputed after the projection)."""
    op = _op('jw')
    gen = torch.Generator().manual_seed(2)
    x0, o = (torch.randn(op.size, dtype=torch.float64, generator=gen).cuda() for _ in range(2))
    o = o / torch.linalg.vector_norm(o)
    op.set_layout(0, 'product')
    got = rq.ground_locg(op, x0, orth=(o,), maxiter=12)
    want = rq.ground_locg(op.matvec, x0, orth=(o,), maxiter=12)
    assert got[0] == want[0] and torch.equal(got[1], want[1])
    e, _, it = rq.ground_locg(op, x0)
    dense = torch.stack([op.matvec(c.contiguous()) for c in
                         torch.eye(op.size, dtype=torch.float64, device='cuda')], 1).cpu().numpy()
    eo, _, ito = OL.ground_locg(lambda v: dense @ v, x0.cpu().numpy())
    assert abs(e - eo) <= 1e-12 * abs(eo) and abs(it - ito) <= 2
