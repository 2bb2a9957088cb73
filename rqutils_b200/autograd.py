r"""Differentiation of the SQD operator and of its ground energy w.r.t. the Pauli coefficients.

Two ``torch.autograd.Function`` s with hand-written backwards:

* :func:`hamiltonian_matvec` — ``y = H(c) v``.  The adjoint w.r.t. ``v`` is ``H^dagger g`` (H is
  Hermitian, so the same CUDA matvec); the adjoint w.r.t. the raw coefficient ``c_r`` is the
  per-term reduction ``Re <g| P_t |v>`` (``sqd_grad_terms``) of the merged term ``t`` that
  ``c_r`` was summed into (PyTorch's conjugate-Wirtinger convention for a real parameter).
* :func:`ground_energy` — ``E0(c)`` from ``ground_locg``; by Hellmann-Feynman
  ``dE0/dc_r = <v0| P_t |v0>`` at the converged, normalised ground vector ``v0``.

The reference has no gradient path (its solver is a ``jax.lax.while_loop``); the only
differentiable object there is the matvec w.r.t. ``PauliSumXZ.c``, which is what these restate.
Raw terms whose coefficient was zero when the Pauli sum was created have no slot in the table
and get zero gradient.  Coefficients are the real raw coefficients (``force_real`` sums).
"""
import contextlib

import torch

from .ground_locg import ground_locg


def _apply_coeffs(op, coeffs):
    """Load ``coeffs`` into the operator's Pauli sum if they differ from the current ones."""
    ham = op.hamiltonian
    c = coeffs.detach().to(torch.float64)
    current, imag = ham.raw_coeffs()
    # coefficients that were set since the operator's last refresh are not in its elements
    if op.coeffs_version != ham.coeffs_version or imag is not None or \
            current.shape != c.shape or not torch.equal(current, c.to(current.device)):
        ham.set_coeffs(c)
        op.refresh()


def _remember(ctx, op):
    """The coefficients a forward pass ran with, for its backward pass."""
    ctx.op = op
    ctx.coeffs = op.hamiltonian.raw_coeffs()[0]    # a copy that no later call writes to
    ctx.version = op.hamiltonian.coeffs_version


@contextlib.contextmanager
def _forward_coeffs(ctx):
    """The operator with the coefficients of the forward pass of ``ctx``; those of a later call
    come back afterwards.  Nothing to do (and no comparison) when none came in between."""
    op, ham = ctx.op, ctx.op.hamiltonian
    if ham.coeffs_version == ctx.version and op.coeffs_version == ctx.version:
        yield op
        return
    (re, im), refreshed = ham.raw_coeffs(), op.coeffs_version == ham.coeffs_version
    _apply_coeffs(op, ctx.coeffs)
    try:
        yield op
    finally:
        ham.set_coeffs(re if im is None else torch.complex(re, im))
        if refreshed:
            op.refresh()


def _scatter_terms(op, g_terms):
    # a gather, not a masked assignment, which would wait for the mask's count on the host
    r2t = op.hamiltonian.raw_to_term()
    return torch.where(r2t >= 0, g_terms[r2t.clamp(min=0)], g_terms.new_zeros(()))


class _Matvec(torch.autograd.Function):
    @staticmethod
    def forward(ctx, coeffs, v, op):
        _apply_coeffs(op, coeffs)
        _remember(ctx, op)
        ctx.save_for_backward(v)
        return op.matvec(v.contiguous())

    @staticmethod
    def backward(ctx, g):
        (v,) = ctx.saved_tensors
        g = g.contiguous()
        gc = gv = None
        with _forward_coeffs(ctx) as op:
            if ctx.needs_input_grad[1]:
                gv = op.matvec(g.to(v.dtype))
            if ctx.needs_input_grad[0]:
                gc = _scatter_terms(op, op.grad_terms(g, v))
        return gc, gv, None


class _GroundEnergy(torch.autograd.Function):
    @staticmethod
    def forward(ctx, coeffs, op, xinit, kwargs):
        _apply_coeffs(op, coeffs)
        e, vec, _ = ground_locg(op, xinit, **kwargs)
        vec = vec / torch.linalg.vector_norm(vec)
        _remember(ctx, op)
        ctx.save_for_backward(vec)
        return torch.tensor(e, dtype=torch.float64, device=vec.device)

    @staticmethod
    def backward(ctx, g):
        (vec,) = ctx.saved_tensors
        with _forward_coeffs(ctx) as op:
            gc = _scatter_terms(op, op.grad_terms(vec, vec)) * g
        return gc, None, None, None


def hamiltonian_matvec(coeffs, v, op):
    """``H(coeffs) @ v`` for an :class:`~rqutils_b200.sqd.SQDOperator`, differentiable in both
    ``coeffs`` (raw real coefficients, one per term the Pauli sum was created from) and ``v``."""
    return _Matvec.apply(coeffs, v, op)


def ground_energy(coeffs, op, xinit=None, **locg_kwargs):
    """Ground energy ``E0(coeffs)`` (0-dim FP64 tensor) with the Hellmann-Feynman gradient.
    ``xinit`` defaults to the operator's ``vinit``; ``locg_kwargs`` go to ``ground_locg``."""
    if xinit is None:
        _apply_coeffs(op, coeffs)
        xinit = op.vinit()
    return _GroundEnergy.apply(coeffs, op, xinit, locg_kwargs)
