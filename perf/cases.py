r"""Performance cases of the SQD path, through the package's public entry points.

Each case is a plain dict (``listed()`` and ``draw()``); ``prepare(case, seed)`` makes what a
program has in hand before the call, ``run(state)`` is one pass, ``work(case)`` the bytes and
operations that a pass cannot do without and ``exact(case, seed)`` the values of its outputs in
64 bits, computed without the package's kernels.

Systems (the package's own workload shapes, seeded):

* ``pauli``: a random Pauli sum on ``n`` qubits (weights 1..4, N(0, 1) coefficients) over
  ``dim`` distinct strings of Hamming weight ``weight``;
* ``jw``: a Jordan-Wigner molecular Hamiltonian of ``norb`` spatial orbitals (2 ``norb`` qubits,
  random integrals with the usual symmetries) over alpha x beta strings of ``nelec`` electrons
  each: all ``na`` x ``nb`` products, or ``dim`` of them drawn at random (``sampled``).
"""
import functools
import itertools
import math

import numpy as np
import torch

import rqutils_b200 as rq
from rqutils_b200.autograd import hamiltonian_matvec
from rqutils_b200.sqd import SQDOperator, Subspace
from rqutils_b200.workloads import labels_from_xz, random_integrals, random_pauli_sum

DTYPES = {'f64': torch.float64, 'c128': torch.complex128, 'f32': torch.float32,
          'c64': torch.complex64}
U64 = np.uint64


def listed():
    return [
        # The smallest matvec: a 16-qubit notebook-sized problem, where the call's latency counts
        # (a caller's own eigensolver or time evolution applies it thousands of times).
        dict(name='matvec_16q_random', kind='matvec', system='pauli', n=16, weight=8, terms=300,
             dim=2000, cache='12', layout='csr', dtype='c128'),
        # The ordinary molecular matvec: 16 orbitals, 512 x 512 product subspace, elements
        # cached, the layout that the package selects for product subspaces.
        dict(name='matvec_32q_product', kind='matvec', system='jw', norb=16, nelec=4, na=512,
             nb=512, cache='12', layout='product', dtype='c128'),
        # The largest: 24 orbitals, 8.7 million rows, in the mixed solver's FP32 precision.
        dict(name='matvec_48q_product_fp32', kind='matvec', system='jw', norb=24, nelec=6,
             na=3072, nb=2816, cache='12', layout='product', dtype='c64'),
        # Determinants sampled from a quantum device, not closed under alpha x beta: ragged
        # rows on the general layout, real vectors (a real Hamiltonian's natural type).
        dict(name='matvec_32q_sampled', kind='matvec', system='jw', norb=16, nelec=4, na=1820,
             nb=1820, sampled=150001, cache='12', layout='csr', dtype='f64'),
        # The reference's default cache strategy (1, 0): sources kept, elements recomputed in
        # every matvec; what a program is left with when the elements do not fit in memory.
        dict(name='matvec_32q_recomputed', kind='matvec', system='jw', norb=16, nelec=4, na=509,
             nb=512, cache='10', layout='csr', dtype='c128'),
        # Nothing kept at all, strategy (0, 0): the largest subspaces for a given memory.
        dict(name='matvec_32q_uncached', kind='matvec', system='jw', norb=16, nelec=4, na=320,
             nb=288, cache='00', layout='csr', dtype='c128'),
        # Building the projected operator of a molecular product subspace, its start index and
        # a first product with it: once per subspace, and an SQD loop visits many.
        dict(name='build_48q_product', kind='build', system='jw', norb=24, nelec=6, na=1152,
             nb=1000, dtype='f64'),
        # The same for a general subspace, where connections are searched pair by pair.
        dict(name='build_40q_random', kind='build', system='pauli', n=40, weight=20, terms=20000,
             dim=131072, dtype='c128'),
        # One step of fitting Pauli coefficients: Hv, its adjoint in both arguments, the
        # coefficients moved along the gradient and Hv again.
        dict(name='grad_32q_product', kind='grad', system='jw', norb=16, nelec=4, na=256, nb=240,
             layout='product', dtype='c128'),
        # The plain FP64 ground-state iteration on a prepared operator (default tolerance).
        dict(name='solve_32q_fp64', kind='solve', system='jw', norb=16, nelec=4, na=448, nb=400,
             layout='product', dtype='f64', maxiter=1000),
        # The whole call from host data: Pauli labels and measured bitstrings with repeats.
        dict(name='sqd_16q_random', kind='sqd', system='pauli', n=16, weight=8, terms=300,
             dim=3000, repeats=500, mode='fp64', vector=True),
        # The whole call on a molecular subspace for its energy alone, mixed precision: one
        # iteration of a self-consistent SQD loop, which keeps the Hamiltonian.
        dict(name='sqd_32q_mixed', kind='sqd', system='jw', norb=16, nelec=4, na=400, nb=360,
             repeats=0, mode='mixed', vector=False),
    ]


def _between(rng, lo, hi):
    """An integer spread evenly over the logarithm of [lo, hi]."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(['matvec', 'matvec', 'matvec', 'matvec', 'build', 'build', 'grad', 'solve',
                       'sqd', 'sqd'])
    if kind == 'matvec':
        cache = rng.choice(['12', '12', '12', '10', '00'])
        which = rng.choice(['pauli', 'jw16', 'jw24', 'sampled'])
        cost = {'12': 1.0, '10': 0.5, '00': 0.3}[cache]
        dtype = rng.choice(['f64', 'c128', 'f32', 'c64'])
        if which == 'pauli':     # odd-Y terms make these Hamiltonians complex
            n = rng.randrange(14, 41)
            cap = min(math.comb(n, n // 2) // 2, int(500000 * cost))
            return dict(kind='matvec', system='pauli', n=n, weight=n // 2,
                        terms=_between(rng, 200, 5000), dim=_between(rng, 1000, cap),
                        cache=cache, layout='csr', dtype=rng.choice(['c128', 'c64']))
        if which == 'sampled':
            return dict(kind='matvec', system='jw', norb=16, nelec=4, na=1820, nb=1820,
                        sampled=_between(rng, 5000, int(150000 * cost)), cache=cache,
                        layout='csr', dtype=dtype)
        norb, nelec = (16, 4) if which == 'jw16' else (24, 6)
        top = (900 if norb == 16 else 2800) * (1.0 if cache == '12' else 0.4)
        return dict(kind='matvec', system='jw', norb=norb, nelec=nelec,
                    na=_between(rng, 60, top), nb=_between(rng, 60, top), cache=cache,
                    layout='product' if cache == '12' else 'csr', dtype=dtype)
    if kind == 'build':
        if rng.random() < 0.4:
            n = rng.randrange(24, 45)
            return dict(kind='build', system='pauli', n=n, weight=n // 2,
                        terms=_between(rng, 1000, 20000), dim=_between(rng, 5000, 131072),
                        dtype='c128')
        norb, nelec = rng.choice([(16, 4), (24, 6)])
        top = 500 if norb == 16 else 1100
        return dict(kind='build', system='jw', norb=norb, nelec=nelec,
                    na=_between(rng, 64, top), nb=_between(rng, 64, top),
                    dtype=rng.choice(['f64', 'c128']))
    if kind == 'grad':
        if rng.random() < 0.4:
            return dict(kind='grad', system='pauli', n=40, weight=20,
                        terms=_between(rng, 1000, 20000), dim=_between(rng, 10000, 200000),
                        layout='csr', dtype='c128')
        return dict(kind='grad', system='jw', norb=16, nelec=4, na=_between(rng, 40, 256),
                    nb=_between(rng, 40, 256), layout=rng.choice(['product', 'csr']),
                    dtype=rng.choice(['f64', 'c128']))
    if kind == 'solve':
        # Capped iterations: a look at the first part of the iteration, as with locg_maxiter.
        return dict(kind='solve', system='jw', norb=16, nelec=4, na=_between(rng, 60, 480),
                    nb=_between(rng, 60, 480), layout=rng.choice(['product', 'csr']),
                    dtype=rng.choice(['f64', 'c128']), maxiter=rng.choice([12, 25]))
    if rng.random() < 0.5:
        n = rng.randrange(12, 21, 2)
        dim = min(_between(rng, 300, 4000), math.comb(n, n // 2) // 2)
        return dict(kind='sqd', system='pauli', n=n, weight=n // 2, terms=_between(rng, 60, 400),
                    dim=dim, repeats=rng.choice([0, dim // 7]), mode='fp64', vector=False)
    return dict(kind='sqd', system='jw', norb=16, nelec=4, na=_between(rng, 64, 400),
                nb=_between(rng, 64, 400), repeats=0, mode=rng.choice(['fp64', 'mixed']),
                vector=False)


# ---------------------------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------------------------
_STRUCTURES = {}


def _parity(v):
    for s in (32, 16, 8, 4, 2, 1):
        v = v ^ (v >> s)
    return v & 1


def _popcount(v, bits):
    c = torch.zeros_like(v)
    for q in range(bits):
        c += (v >> q) & 1
    return c


def _ladder_terms(ops, col, weight, nq):
    """X^x Z^z monomials (x, z, column, weight) of products of ladder operators; ``ops`` lists
    (orbital indices, dagger) from left to right.  A ladder operator on qubit p is
    X_p Z_{<p} (1 -/+ Z_p) / 2; the weights are signed powers of two, so sums of them are exact."""
    out = []
    for combo in range(1 << len(ops)):
        x = torch.zeros_like(col)
        z = torch.zeros_like(col)
        w = torch.full(col.shape, weight, dtype=torch.float64, device=col.device)
        for k, (idx, dagger) in enumerate(ops):
            e = torch.ones_like(idx) << idx
            with_z = (combo >> k) & 1
            w = w * (1 - 2 * ((z & e) != 0).double())
            w = w * (0.5 if (not with_z or dagger) else -0.5)
            x = x ^ e
            z = z ^ ((e - 1) | e if with_z else e - 1)
        # X^x Z^z = (-i)^{|x & z|} Q(x, z); imaginary parts cancel in the sum
        ph = _popcount(x & z, nq) & 3
        w = torch.where(ph == 0, w, torch.where(ph == 2, -w, torch.zeros_like(w)))
        keep = w != 0
        out.append((x[keep], z[keep], col[keep], w[keep]))
    return out


def _merge_terms(x, z, col, w):
    for k in (2, 1, 0):                # ascending (x, z, column)
        o = torch.sort((x, z, col)[k], stable=True).indices
        x, z, col, w = x[o], z[o], col[o], w[o]
    new = torch.ones_like(x, dtype=torch.bool)
    new[1:] = (x[1:] != x[:-1]) | (z[1:] != z[:-1]) | (col[1:] != col[:-1])
    seg = torch.cumsum(new, 0) - 1
    s = torch.zeros(int(seg[-1]) + 1, dtype=torch.float64, device=x.device).index_add_(0, seg, w)
    live = s != 0                      # sums of signed powers of two: exact
    return x[new][live], z[new][live], col[new][live], s[live]


def _jw_structure(norb):
    """Pauli masks of the Jordan-Wigner Hamiltonian of ``norb`` orbitals and the linear map from
    its integrals to their coefficients (the same for all seeds)."""
    if norb in _STRUCTURES:
        return _STRUCTURES[norb]
    dev = 'cuda'
    nq = 2 * norb
    r = torch.arange(norb, device=dev)
    s2 = torch.arange(2, device=dev)
    i, j, s = (t.reshape(-1) for t in torch.meshgrid(r, r, s2, indexing='ij'))
    parts = _ladder_terms([(i + norb * s, True), (j + norb * s, False)], i * norb + j, 1.0, nq)
    i, j, k, l, s, t = (a.reshape(-1) for a in torch.meshgrid(r, r, r, r, s2, s2, indexing='ij'))
    p, q, v, u = i + norb * s, k + norb * t, l + norb * t, j + norb * s
    keep = (p != q) & (v != u)
    a, b = torch.minimum(i, j) * norb + torch.maximum(i, j), \
        torch.minimum(k, l) * norb + torch.maximum(k, l)
    col = norb ** 2 + torch.minimum(a, b) * norb ** 2 + torch.maximum(a, b)
    p, q, v, u, col = (m[keep] for m in (p, q, v, u, col))
    step = 1 << 18
    for o in range(0, p.shape[0], step):
        c = slice(o, o + step)
        parts.append(_merge_terms(*(torch.cat(m) for m in zip(*_ladder_terms(
            [(p[c], True), (q[c], True), (v[c], False), (u[c], False)], col[c], 0.5, nq)))))
    x, z, col, w = (m.cpu().numpy() for m in
                    _merge_terms(*(torch.cat(m) for m in zip(*parts))))
    new = np.concatenate([[True], (x[1:] != x[:-1]) | (z[1:] != z[:-1])])
    _STRUCTURES[norb] = (x[new].view(U64), z[new].view(U64), np.nonzero(new)[0], col, w)
    torch.cuda.empty_cache()
    return _STRUCTURES[norb]


def _hamiltonian(case, rng):
    """(x masks, z masks, real coefficients, qubits)."""
    if case['system'] == 'pauli':
        x, z, c = random_pauli_sum(case['n'], case['terms'], rng,
                                   scale=1.0 / math.sqrt(case['terms']))
        return x, z, c, case['n']
    norb = case['norb']
    x, z, start, col, w = _jw_structure(norb)
    h1, h2 = random_integrals(norb, rng)
    flat = np.concatenate([h1.reshape(-1), h2.reshape(-1)])
    c = np.add.reduceat(w * flat[col], start)
    keep = np.abs(c) > 1e-12
    return x[keep], z[keep], c[keep], 2 * norb


@functools.lru_cache(maxsize=None)
def _all_strings(n, k):
    return np.array([sum(1 << q for q in c) for c in itertools.combinations(range(n), k)],
                    dtype=U64)


def _weight_strings(n, k, d, rng):
    """``d`` distinct ``n``-bit strings of weight ``k``, ascending."""
    if math.comb(n, k) <= 1 << 18:
        return np.sort(rng.choice(_all_strings(n, k), size=d, replace=False))
    gen = torch.Generator(device='cuda')
    gen.manual_seed(int(rng.integers(1 << 40)))
    got = torch.zeros(0, dtype=torch.int64, device='cuda')
    while got.shape[0] < d:
        keys = torch.rand((d + d // 8 + 16, n), generator=gen, device='cuda')
        at = torch.topk(keys, k, dim=1).indices
        got = torch.unique(torch.cat([got, (torch.ones_like(at) << at).sum(1)]))
    drop = torch.randperm(got.shape[0], generator=gen, device='cuda')[:d]
    return torch.sort(got[drop]).values.cpu().numpy().view(U64)


def _states(case, rng):
    if case['system'] == 'pauli':
        return _weight_strings(case['n'], case['weight'], case['dim'], rng)
    norb, nelec = case['norb'], case['nelec']
    alpha = _weight_strings(norb, nelec, case['na'], rng)
    beta = _weight_strings(norb, nelec, case['nb'], rng)
    states = ((beta[:, None] << U64(norb)) | alpha[None, :]).reshape(-1)
    if 'sampled' in case:
        states = np.sort(rng.choice(states, size=case['sampled'], replace=False))
    return states


def _bits(states, n):
    shifts = np.arange(n - 1, -1, -1, dtype=U64)
    return ((states[:, None] >> shifts[None, :]) & U64(1)).astype(np.uint8)


def _inputs(case, seed):
    rng = np.random.default_rng(seed)
    x, z, c, n = _hamiltonian(case, rng)
    return rng, x, z, c, n, _states(case, rng)


def _vector(count, dtype, seed):
    gen = torch.Generator(device='cuda')
    gen.manual_seed(int(seed) + 7919)
    v = torch.randn(count, dtype=dtype, generator=gen, device='cuda')
    return v / torch.linalg.vector_norm(v)


def _operator(case, x, z, c, n, states):
    ham = rq.PauliSumXZ.from_xz(x, z, c, n, force_real=True, padded=True)
    space = Subspace.from_u64(states, n)
    op = SQDOperator(ham, space, cache_strategy=tuple(int(d) for d in case.get('cache', '12')))
    if case['layout'] != 'csr':
        op.set_layout(0, case['layout'])
        op.set_layout(1, case['layout'])
    return op


def prepare(case, seed):
    rng, x, z, c, n, states = _inputs(case, seed)
    kind = case['kind']
    if kind == 'build':
        space = Subspace.from_u64(states, n)
        return dict(kind=kind, space=space,
                    v=_vector(space.states_size, DTYPES[case['dtype']], seed),
                    ham=rq.PauliSumXZ.from_xz(x, z, c, n, force_real=True, padded=True))
    if kind == 'sqd':
        more = rng.choice(states, size=case['repeats'])
        bits = _bits(rng.permutation(np.concatenate([states, more])), n)
        if case['system'] == 'jw':   # the loop over subspaces keeps its Hamiltonian
            ham = rq.PauliSumXZ.from_xz(x, z, c, n, force_real=True, padded=True)
        else:
            ham = (labels_from_xz(x, z, n), list(c))
        return dict(kind=kind, ham=ham, bits=bits,
                    options=dict(return_eigvec=case['vector'], locg_mode=case['mode']))
    op = _operator(case, x, z, c, n, states)
    dtype = DTYPES[case['dtype']]
    v = _vector(op.size, dtype, seed)
    if kind == 'matvec':
        return dict(kind=kind, op=op, v=v, out=torch.empty_like(v))
    if kind == 'solve':
        return dict(kind=kind, op=op, v=v, maxiter=case['maxiter'])
    return dict(kind=kind, op=op, v=v.requires_grad_(True),
                g=_vector(op.size, dtype, seed + 1),
                coeffs=torch.as_tensor(c, device='cuda').requires_grad_(True))


def run(state):
    kind = state['kind']
    if kind == 'matvec':
        return state['op'].matvec(state['v'], state['out'])
    if kind == 'build':
        op = SQDOperator(state['ham'], state['space'], cache_strategy=(1, 2))
        return op.vinit(), op.matvec(state['v'])
    if kind == 'sqd':
        return rq.sqd(state['ham'], state['bits'], options=state['options'])
    if kind == 'solve':
        energy, vec, _ = rq.ground_locg(state['op'], state['v'], maxiter=state['maxiter'])
        return energy, vec
    coeffs, v, op = state['coeffs'], state['v'], state['op']
    y = hamiltonian_matvec(coeffs, v, op)
    gc, gv = torch.autograd.grad(y, (coeffs, v), state['g'])
    with torch.no_grad():
        moved = coeffs - 0.1 * gc
        again = hamiltonian_matvec(moved, v, op)
    return y.detach(), gc, gv, moved, again


# ---------------------------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------------------------
def _size(case):
    """(rows, stored pairs, terms, groups) expected on average."""
    if case['system'] == 'pauli':
        n, k, d, m = case['n'], case['weight'], case['dim'], case['terms']
        per = 0.0
        for w in range(1, 5):
            for b in range(0, w + 1):            # b of the w letters flip their qubit
                p = 0.25 * math.comb(w, b) * (2 / 3) ** b * (1 / 3) ** (w - b)
                if b == 0 or b % 2:
                    continue
                stay = math.comb(b, b // 2) * math.comb(n - b, k - b // 2) / math.comb(n, k)
                per += m * p * stay * d / math.comb(n, k)
        return d, d * (1 + per), m, 0.85 * m
    norb, ne = case['norb'], case['nelec']
    s = ne * (norb - ne)
    two = math.comb(ne, 2) * math.comb(norb - ne, 2)
    total = math.comb(norb, ne)
    terms, groups = {16: (94849, 18281), 24: (485281, 97981)}[norb]
    fa, fb = case['na'] / total, case['nb'] / total
    rows = case['na'] * case['nb']
    keep = 1.0
    if 'sampled' in case:
        keep = case['sampled'] / rows
        rows = case['sampled']
    return rows, rows * (1 + keep * ((s + two) * (fa + fb) + s * s * fa * fb)), terms, groups


def work(case):
    rows, pairs, terms, groups = _size(case)
    cx = case['system'] == 'pauli'               # odd-Y terms: complex elements
    kind = case['kind']
    table = 24 * terms + 16 * groups
    per_pair = terms / groups                    # terms of an element, on average
    dtype = DTYPES[case.get('dtype', 'c128')]
    wv = dtype.itemsize
    elem = (16 if cx else 8) // (2 if dtype in (torch.float32, torch.complex64) else 1)
    fma = 2 * (2 if cx else 1) * (2 if dtype.is_complex else 1)
    one = dict(bytes=2 * rows * wv, flops=pairs * fma)      # one matvec
    cache = case.get('cache', '12')
    if cache == '12':
        one['bytes'] += pairs * elem
    else:
        one['bytes'] += 8 * rows + table + (4 * pairs if cache == '10' else 0)
        one['flops'] += pairs * per_pair
    if kind == 'matvec':
        return one
    if kind == 'build':
        # states and Pauli table in; row offsets, columns and elements out; then one product
        return dict(bytes=one['bytes'] + 16 * rows + table + pairs * (elem + 4),
                    flops=one['flops'] + pairs * per_pair)
    if kind == 'grad':
        # Hv, H g, the per-term sums over all pairs, new elements and Hv again
        return dict(bytes=3 * one['bytes'] + pairs * (elem + 4) + 2 * rows * wv + 2 * table,
                    flops=3 * one['flops'] + 2 * pairs * per_pair)
    # a solve: three products and about forty vector reads or writes per iteration
    iters = min(case.get('maxiter', 1000), 40 if case.get('mode') == 'mixed' else 150)
    per = 1 if case.get('mode') == 'mixed' else 3
    build = 12 * pairs + table if kind == 'sqd' else 0
    return dict(bytes=build + iters * (per * one['bytes'] + 33 * rows * wv),
                flops=iters * (per * one['flops'] + 60 * rows * wv / 8))


# ---------------------------------------------------------------------------------------------
# The same in 64 bits, in plain torch
# ---------------------------------------------------------------------------------------------
class _Plain:
    """H on the subspace group by group: for each X mask the rows with a source, their sources
    and the composed diagonal (a real or complex element per row)."""

    def __init__(self, x, z, c, states):
        order = np.lexsort((z, x))
        self.order = order
        x, z, c = x[order], z[order], c[order]
        ph = np.bitwise_count(x & z).astype(np.int64) & 3
        self.phase = torch.as_tensor(np.array([1, -1j, -1, 1j])[ph], device='cuda')
        self.c = torch.as_tensor(c, device='cuda')
        self.z = torch.as_tensor(z.view(np.int64), device='cuda')
        self.real = not np.any(ph & 1)
        self.starts = np.nonzero(np.concatenate([[True], x[1:] != x[:-1]]))[0]
        self.ends = np.append(self.starts[1:], x.shape[0])
        self.gx = [int(v) for v in x[self.starts]]
        self.states = torch.as_tensor(states.view(np.int64), device='cuda')

    def groups(self):
        s = self.states
        for x, b, e in zip(self.gx, self.starts, self.ends):
            if x == 0:
                rows = src = torch.arange(s.shape[0], device='cuda')
            else:
                want = s ^ x
                at = torch.searchsorted(s, want).clamp_(max=s.shape[0] - 1)
                rows = torch.nonzero(s[at] == want).flatten()
                src = at[rows]
            if rows.shape[0]:
                yield rows, src, int(b), int(e)

    def signs(self, rows, b, e):
        """(-1)^{|s & z|} of the rows for terms b..e, blocks of rows at a time."""
        step = max(1, (1 << 24) // (e - b))
        for o in range(0, rows.shape[0], step):
            r = rows[o:o + step]
            yield slice(o, o + step), \
                1.0 - 2.0 * _parity(self.states[r][:, None] & self.z[None, b:e]).double()

    def coefficients(self, c=None):
        t = (self.c if c is None else c) * self.phase
        return t.real.clone() if self.real else t

    def apply(self, vs, cs, grad=None):
        """H(c) v for each (v, c); with ``grad`` = (u, v) also Re <u| P_t |v> of every term."""
        outs = [torch.zeros(v.shape, dtype=torch.promote_types(v.dtype, c.dtype), device='cuda')
                for v, c in zip(vs, cs)]
        g = None if grad is None else torch.zeros(self.z.shape[0], dtype=torch.float64,
                                                  device='cuda')
        for rows, src, b, e in self.groups():
            for part, sg in self.signs(rows, b, e):
                r, q = rows[part], src[part]
                for out, v, c in zip(outs, vs, cs):
                    el = sg.to(c.dtype) @ c[b:e]
                    out[r] += el * v[q]
                if g is not None:
                    w = grad[0][r].conj() * grad[1][q]
                    if w.is_complex():
                        g[b:e] += ((sg.T.to(w.dtype) @ w) * self.phase[b:e]).real
                    else:
                        g[b:e] += (sg.T @ w) * self.phase[b:e].real
        return outs, g

    def dense(self):
        n = self.states.shape[0]
        c = self.coefficients()
        h = torch.zeros((n, n), dtype=c.dtype, device='cuda')
        for rows, src, b, e in self.groups():
            for part, sg in self.signs(rows, b, e):
                h[rows[part], src[part]] += sg.to(c.dtype) @ c[b:e]
        return h


def exact(case, seed):
    kind = case['kind']
    rows, pairs, terms, groups = _size(case)
    if kind in ('solve', 'sqd'):
        if rows > 4500 or case.get('maxiter', 1000) < 1000:
            return None
        _, x, z, c, n, states = _inputs(case, seed)
        e = float(torch.linalg.eigvalsh(_Plain(x, z, c, states).dense())[0])
        return ((e, None) if kind == 'solve' else (e, None, None) if case['vector'] else e)
    if rows * groups > 6e9:
        return None
    _, x, z, c, n, states = _inputs(case, seed)
    plain = _Plain(x, z, c, states)
    wide = torch.complex128 if DTYPES[case['dtype']].is_complex else torch.float64
    v = _vector(rows, DTYPES[case['dtype']], seed).to(wide)
    cf = plain.coefficients()
    if kind in ('matvec', 'build'):
        hv = plain.apply([v], [cf])[0][0]
        return hv if kind == 'matvec' else (None, hv)
    g = _vector(rows, DTYPES[case['dtype']], seed + 1).to(wide)
    (y, gv), gt = plain.apply([v, g], [cf, cf], grad=(g, v))
    gc = torch.zeros(x.shape[0], dtype=torch.float64, device='cuda')
    at = torch.as_tensor(plain.order, device='cuda')
    gc[at] = gt                      # repeated Pauli strings each get their string's derivative
    moved = torch.as_tensor(c, device='cuda') - 0.1 * gc
    (again,), _ = plain.apply([v], [plain.coefficients(moved[at])])
    return y, gc, gv, moved, again
