"""Per-term sums Re <u| P_t |v> on product and general subspaces, with groups longer than a block's
64 terms and two-half groups longer than a warp's eight, against a NumPy sum per term."""
import numpy as np
import pytest
import torch

import rqutils_b200 as rq
from rqutils_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _case(name):
    rng = np.random.default_rng(6)
    if name.startswith('jw'):
        na, nb = {'jw': (37, 33), 'jw-one-low': (1, 40), 'jw-sampled': (37, 33)}[name]
        wl = W.jw_workload(name, 8, 3, na, nb, 5)
        states = wl.states
        if name == 'jw-sampled':
            states = np.sort(rng.choice(states, size=701, replace=False))
        return wl.x, wl.z, wl.coeffs, states, 16, True
    # groups of 1..130 terms on each class of masks, complex elements; 1,100 rows: two tiles
    masks = np.array([0, 3, 5, 0x300, 0x900, 0x303, 0x905, 0x50c], dtype=np.uint64)
    counts = [150, 65, 1, 130, 64, 17, 8, 9]
    x = np.repeat(masks, counts)
    z = np.concatenate([rng.choice(1 << 12, size=k, replace=False).astype(np.uint64)
                        for k in counts])
    c = rng.standard_normal(x.shape[0])
    if name == 'long-no-diagonal':
        x, z, c = x[150:], z[150:], c[150:]
    hi = np.sort(rng.choice(64, size=44, replace=False)).astype(np.uint64)
    lo = np.sort(rng.choice(64, size=25, replace=False)).astype(np.uint64)
    return x, z, c, ((hi[:, None] << np.uint64(6)) | lo[None, :]).reshape(-1), 12, False


@pytest.mark.parametrize('name', ['jw', 'jw-one-low', 'jw-sampled', 'long', 'long-no-diagonal'])
def test_grad_terms(name):
    x, z, c, states, n, real = _case(name)
    ham = rq.PauliSumXZ.from_xz(x, z, c, n, force_real=real, padded=True)
    op = rq.SQDOperator(ham, rq.Subspace.from_u64(states, n), cache_strategy=(1, 2))
    gx, gs, tz, _, _ = (t.cpu().numpy() for t in ham.device_tables())
    gx, tz = gx.view(np.uint64), tz.view(np.uint64)
    for dt in ([torch.float64, torch.complex128] if real else [torch.complex128]):
        u, v = (torch.randn(op.size, dtype=dt, device='cuda') for _ in range(2))
        un, vn = u.cpu().numpy(), v.cpu().numpy()
        want = np.zeros(tz.shape[0])
        scale = np.zeros(tz.shape[0])
        for j, xm in enumerate(gx):
            src = states ^ xm
            at = np.minimum(np.searchsorted(states, src), states.shape[0] - 1)
            r = np.nonzero(states[at] == src)[0]
            w = un[r].conj() * vn[at[r]]
            for t in range(gs[j], gs[j + 1]):
                sign = 1.0 - 2.0 * (np.bitwise_count(states[r] & tz[t]) & 1)
                ph = (-1j) ** int(np.bitwise_count(xm & tz[t]))
                want[t] = (ph * sign * w).real.sum()
                scale[t] = np.abs(w).sum()
        got = op.grad_terms(u, v).cpu().numpy()
        # at most states.size terms in a sum, each rounded by a few ulps
        bound = 4 * np.finfo(float).eps * np.sqrt(states.shape[0]) * np.maximum(scale, 1e-300)
        assert (np.abs(got - want) <= bound + 1e-300).all()
        assert torch.equal(op.grad_terms(u, v)[1:2], op.grad_terms(u, v)[1:2])
