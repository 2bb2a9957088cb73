"""Backward passes run with the coefficients of their own forward pass, whatever was set in between,
and leave the operator as they found it; against dense matrices."""
import numpy as np
import pytest
import torch

import rqutils_b200 as rq
from rqutils_b200 import workloads as W
from rqutils_b200.autograd import hamiltonian_matvec, ground_energy
from oracle import dense as OD

pytestmark = pytest.mark.gpu
N = 10


def _case(cache):
    rng = np.random.default_rng(11)
    x, z, c = W.random_pauli_sum(N, 40, rng, scale=0.5)
    states = W.weight_subspace(N, 5, 120, rng)
    ham = rq.PauliSumXZ.from_xz(x, z, c, N, force_real=True, padded=True)
    op = rq.SQDOperator(ham, rq.Subspace.from_u64(states, N), cache_strategy=cache)
    labels = W.labels_from_xz(x, z, N)

    def dense(coeffs):
        return torch.as_tensor(OD.projected_matrix(labels, coeffs, states))
    terms = [dense_term(labels[k], states) for k in range(len(c))]
    return ham, op, c, dense, terms


def dense_term(label, states):
    return torch.as_tensor(OD.projected_matrix([label], [1.0], states))


def _vectors(op):
    gen = torch.Generator().manual_seed(3)
    return [torch.randn(op.size, dtype=torch.complex128, generator=gen) for _ in range(3)]


@pytest.mark.parametrize('cache', [(1, 0), (1, 2)])
def test_two_forwards_before_one_backward(cache):
    ham, op, c, dense, terms = _case(cache)
    cs = [torch.as_tensor(k, device='cuda').requires_grad_(True) for k in (c, 0.3 * c + 0.2)]
    v, g1, g2 = _vectors(op)
    vs = [v.cuda().requires_grad_(True) for _ in cs]
    ys = [hamiltonian_matvec(k, u, op) for k, u in zip(cs, vs)]
    torch.autograd.backward(ys, [g1.cuda(), g2.cuda()])
    for k, u, g in zip(cs, vs, (g1, g2)):
        ref = dense(k.detach().cpu().numpy()) @ g
        assert (u.grad.cpu() - ref).abs().max() <= 1e-12 * ref.abs().max()
        want = torch.stack([torch.vdot(g, t @ v).real for t in terms])
        assert (k.grad.cpu() - want).abs().max() <= 1e-12 * want.abs().max()
    # the operator still holds the last coefficients
    ref = dense(cs[1].detach().cpu().numpy()) @ v
    assert (op.matvec(v.cuda()).cpu() - ref).abs().max() <= 1e-12 * ref.abs().max()


@pytest.mark.parametrize('cache', [(1, 0), (1, 2)])
def test_coefficients_set_elsewhere(cache):
    """Set on the Pauli sum between forward and backward, and by a second operator on it."""
    ham, op, c, dense, _ = _case(cache)
    other = rq.SQDOperator(ham, op.space, cache_strategy=cache)
    k = torch.as_tensor(c, device='cuda')
    v, g, _ = _vectors(op)
    u = v.cuda().requires_grad_(True)
    y = hamiltonian_matvec(k, u, op)
    ham.set_coeffs(-k)
    op.refresh()
    y.backward(g.cuda())
    ref = dense(c) @ g
    assert (u.grad.cpu() - ref).abs().max() <= 1e-12 * ref.abs().max()
    assert (op.matvec(g.cuda()).cpu() + ref).abs().max() <= 1e-12 * ref.abs().max()
    # the same coefficients again, after the other operator loaded its own
    hamiltonian_matvec(k, u, op)
    hamiltonian_matvec(2 * k, u, other)
    ref = dense(c) @ v
    assert (hamiltonian_matvec(k, u, op).detach().cpu() - ref).abs().max() <= \
        1e-12 * ref.abs().max()


def test_energy_gradient_after_other_coefficients():
    ham, op, c, dense, terms = _case((1, 2))
    k = torch.as_tensor(c, device='cuda').requires_grad_(True)
    e = ground_energy(k, op)
    zero = c.copy()
    zero[::2] = 0.0                 # a zero ends its group's sums
    ground_energy(torch.as_tensor(zero, device='cuda'), op)
    e.backward()
    w, u = np.linalg.eigh(dense(c).numpy())
    x = torch.as_tensor(u[:, 0])
    want = torch.stack([torch.vdot(x, t @ x).real for t in terms])
    # first order in the vector's error, the default residual over the gap
    assert (k.grad.cpu() - want).abs().max() <= 1e-6
