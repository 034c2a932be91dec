"""Performance cases of the block-sparse tensor backend.

Each case is one call sequence that YASTN's tensor, MPS or PEPS layer issues: a tensordot
(transpose_and_merge of both operands, the sector products, unmerge), a pure fuse of legs, a
truncated SVD (svd, fix_svd_signs, truncation, apply_mask), a QR, a Hermitian
eigendecomposition, or a Lanczos expansion of the DMRG two-site effective Hamiltonian. The
metadata tuples have the formats of YASTN's metadata layer and are built once per structure, as
YASTN memoises them.
"""
import functools
import itertools
import math

import numpy as np
import torch

from yastn_gb300 import backend, krylov, ops
from yastn_gb300.workloads import Heff2Workload, load_trace

TOL = 1e-12  # relative cut of the truncated SVDs: below it only rounding noise
DTYPES = {'f64': torch.float64, 'c128': torch.complex128, 'f32': torch.float32}


# ----------------------------------------------------------------------------- the cases

def listed():
    return [
        # MPS tensors of a spin-1 chain at a small bond dimension: launches and host latency
        dict(name='tensordot_small', kind='tensordot', D1=16, w1=3, D2=3, w2=1, dtype='f64', mode='fp64', grad=False),
        # an MPS-sized contraction inside an optimisation: forward and both adjoints
        dict(name='tensordot_grad', kind='tensordot', D1=301, w1=5, D2=3, w2=1, dtype='f64', mode='fp64', grad=True),
        # the U(1) D = 64 rank-4 benchmark contraction, 13 sectors up to about 850, on the tensor cores
        dict(name='tensordot_emulated', kind='tensordot', D1=64, w1=3, D2=64, w2=3, dtype='f64', mode='emulated',
             grad=False),
        # fusing the legs of a large rank-5 tensor with odd extents, and its adjoint
        dict(name='fuse_grad', kind='fuse', D=45, w=1, order='41302', split=2, dtype='f64', grad=True),
        # the truncated SVD of a two-site DMRG update at a small bond dimension
        dict(name='svd_small', kind='svd', D=32, w=3, decades=8, noise=False, dtype='f64', keep=0.5, ratio=1.0,
             grad=False),
        # the same at a bond dimension of several hundred: sectors up to about 140
        dict(name='svd_dmrg', kind='svd', D=513, w=4, decades=8, noise=False, dtype='f64', keep=0.5, ratio=1.0,
             grad=False),
        # the projector SVD of an iPEPS corner transfer matrix step (Z2, D = 6, chi = 24: 2 blocks of
        # 432): a spectrum over many decades with a tail of rounding noise, of which chi values are kept
        dict(name='svd_ctm', kind='svd', D=864, w=0, decades=9, noise=True, dtype='f64', keep=0.03, ratio=1.0,
             grad=False),
        # the same at chi = 72
        dict(name='svd_ctm_large', kind='svd', D=2592, w=0, decades=9, noise=True, dtype='f64', keep=0.028,
             ratio=1.0, grad=False),
        # a complex SVD inside a differentiated network: rectangular sectors, forward and adjoint
        dict(name='svd_c128_grad', kind='svd', D=200, w=2, decades=4, noise=False, dtype='c128', keep=0.4, ratio=1.3,
             grad=True),
        # QR projectors of a differentiated corner transfer matrix step: forward and adjoint
        dict(name='qr_grad', kind='qr', D=864, w=0, ratio=1.25, dtype='f64', grad=True),
        # Hermitian eigendecomposition of a density matrix's sectors
        dict(name='eigh', kind='eigh', D=401, w=2, dtype='f64'),
        # DMRG's inner loop: Lanczos on the two-site effective Hamiltonian (XXZ, D = 1024)
        dict(name='lanczos_heff2', kind='lanczos', ncv=16, mode='emulated'),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(('tensordot', 'tensordot', 'tensordot', 'fuse', 'svd', 'svd', 'svd', 'qr', 'eigh', 'lanczos'))
    if kind == 'tensordot':
        if rng.random() < 0.5:  # MPS tensors: a long leg and a physical one
            d1, w1, d2, w2 = _log_int(rng, 16, 400), rng.randint(2, 6), rng.randint(2, 5), rng.randint(0, 1)
            d2 = max(d2, 2 * w2 + 1)
        else:                   # PEPS-like tensors: legs of similar extents
            d1, w1 = _log_int(rng, 8, 60), rng.randint(1, 3)
            d2, w2 = _log_int(rng, 8, 60), rng.randint(1, 3)
        return dict(kind=kind, D1=max(d1, 2 * w1 + 1), w1=w1, D2=max(d2, 2 * w2 + 1), w2=w2,
                    dtype=rng.choice(('f64', 'f64', 'c128')), mode=rng.choice(('fp64', 'fp64', 'emulated')),
                    grad=rng.random() < 0.4)
    if kind == 'fuse':
        order = list('01234')
        rng.shuffle(order)
        w = rng.randint(0, 2)
        return dict(kind=kind, D=max(_log_int(rng, 4, 44), 2 * w + 1), w=w, order=''.join(order),
                    split=rng.randint(1, 4), dtype=rng.choice(('f64', 'f64', 'c128', 'f32')), grad=rng.random() < 0.5)
    if kind == 'svd':
        cplx = rng.random() < 0.3
        w = rng.randint(0, 4)
        noise = not cplx and rng.random() < 0.4
        grad = not noise and rng.random() < 0.4
        return dict(kind=kind, D=_log_int(rng, 16 * (w + 1), 400 if cplx else 1000), w=w,
                    decades=rng.randint(2, 4) if grad else rng.randint(4, 9), noise=noise,
                    dtype='c128' if cplx else 'f64', keep=round(rng.uniform(0.02, 0.1 if noise else 0.5), 3),
                    ratio=round(rng.uniform(0.6, 1.7), 2), grad=grad)
    if kind == 'qr':
        w = rng.randint(0, 4)
        return dict(kind=kind, D=_log_int(rng, 16 * (w + 1), 860), w=w, ratio=round(rng.uniform(1.1, 2.0), 2),
                    dtype=rng.choice(('f64', 'f64', 'c128')), grad=rng.random() < 0.5)
    if kind == 'eigh':
        w = rng.randint(0, 4)
        return dict(kind=kind, D=_log_int(rng, 16 * (w + 1), 400), w=w, dtype=rng.choice(('f64', 'f64', 'c128')))
    return dict(kind=kind, ncv=rng.randint(2, 15), mode=rng.choice(('fp64', 'emulated')))


# ----------------------------------------------------------------------------- structures

def _leg(D, w):
    """{charge: dimension} over -w..w with a bell-shaped distribution of total dimension D."""
    g = [math.exp(-0.5 * (2.0 * t / (w + 1)) ** 2) for t in range(-w, w + 1)]
    dims = [max(1, int(D * x / sum(g))) for x in g]
    dims[w] += D - sum(dims)
    return {t: d for t, d in zip(range(-w, w + 1), dims) if d > 0}


def _prod(xs):
    return math.prod(xs)


def _layout(items):
    """Consecutive slices for {charge: block shape}."""
    out, low = {}, 0
    for t, D in items:
        out[t] = ((low, low + _prod(D)), D)
        low += _prod(D)
    return out, low


class _Fused:
    """A tensor whose legs, reordered by ``order``, are fused into groups: its blocks, the fused
    blocks, and the metadata of transpose_and_merge and of unmerge (of the reordered legs)."""

    def __init__(self, legs, signs, order, groups):
        charges = [c for c in itertools.product(*legs) if sum(s * t for s, t in zip(signs, c)) == 0]
        self.blocks, self.size = _layout([(c, tuple(l[t] for l, t in zip(legs, c))) for c in charges])
        self.order = tuple(order)

        def eff(t, group):
            return sum(signs[i] * t[i] for i in group)
        self.fused_of = {c: tuple(eff(c, g) for g in groups) for c in charges}
        spans = []  # per group: {fused charge: {leg charges: (start, stop)}}
        for gi, g in enumerate(groups):
            sp = {}
            for sub in sorted({tuple(c[i] for i in g) for c in charges}):
                q = sum(signs[i] * t for i, t in zip(g, sub))
                at = sp.setdefault(q, {})
                low = max((b for _, b in at.values()), default=0)
                at[sub] = (low, low + _prod(legs[i][t] for i, t in zip(g, sub)))
            spans.append(sp)
        new = sorted(set(self.fused_of.values()))
        dims = {q: tuple(max(b for _, b in spans[gi][q[gi]].values()) for gi in range(len(groups))) for q in new}
        self.new, self.new_size = _layout([(q, dims[q]) for q in new])
        self.meta_new = tuple((q, D, sl) for q, (sl, D) in self.new.items())
        mrg, um, low = [], [], 0
        for c in sorted(charges, key=lambda c: (self.fused_of[c], c)):
            sl, D = self.blocks[c]
            q = self.fused_of[c]
            sub = tuple(spans[gi][q[gi]][tuple(c[i] for i in g)] for gi, g in enumerate(groups))
            mrg.append((q, sl, D, sub, tuple(b - a for a, b in sub)))
            Dt = tuple(D[i] for i in self.order)
            um.append(((low, low + _prod(Dt)), Dt, self.new[q][0], self.new[q][1], sub))
            low += _prod(Dt)
        self.meta_mrg, self.meta_unmerge = tuple(mrg), tuple(um)


@functools.lru_cache(maxsize=64)
def _tensordot_structure(D1, w1, D2, w2):
    """A[x1 k1 x2 k2] B[k1 y1 k2 y2] = C[x1 x2 y1 y2]; fused A (x1 x2 | k1 k2), B (k1 k2 | y1 y2)."""
    l1, l2 = _leg(D1, w1), _leg(D2, w2)
    legs, signs, order = (l1, l1, l2, l2), (1, -1, 1, -1), (0, 2, 1, 3)
    op = _Fused(legs, signs, order, ((0, 2), (1, 3)))  # A and B have the same structure
    c = _Fused((l1, l2, l1, l2), (1, 1, -1, -1), (0, 1, 2, 3), ((0, 1), (2, 3)))
    dot = tuple((c.new[q][0], c.new[q][1], sl, D, sl, D) for q, (sl, D) in op.new.items())
    return op, c, dot


@functools.lru_cache(maxsize=64)
def _fuse_structure(D, w, order, split):
    legs = [_leg(max(2 * w + 1, D - 2 * i), w) for i in range(5)]
    order = tuple(int(c) for c in order)
    return _Fused(legs, (1, 1, 1, -1, -1), order, (order[:split], order[split:]))


@functools.lru_cache(maxsize=64)
def _matrix_structure(D, w, ratio):
    """Sectors (m x n) of a matrix of total column dimension D, m = ratio n; w = 0: two equal
    sectors (Z2). Returns the svd, qr and eigh records and the flat sizes."""
    if w == 0:
        cols = {0: D - D // 2, 1: D // 2}
    else:
        cols = _leg(D, w)
    svd, qr, eigh = [], [], []
    a = u = s = v = r = q = 0
    for t, n in cols.items():
        m = max(1, round(ratio * n))
        k = min(m, n)
        rec = ((a, a + m * n), (m, n), (u, u + m * k), (m, k), (s, s + k), (v, v + k * n), (k, n))
        svd.append(rec)
        qr.append((rec[0], (m, n), (q, q + m * k), (m, k), (r, r + k * n), (k, n)))
        eigh.append(((a, a + n * n), (n, n), (a, a + n * n), (n, n), (s, s + n)))
        a, u, s, v, q, r = a + m * n, u + m * k, s + k, v + k * n, q + m * k, r + k * n
    return dict(svd=tuple(svd), qr=tuple(qr), eigh=tuple(eigh), size=a, svd_sizes=(u, s, v), qr_sizes=(q, r),
                eigh_sizes=(s, a))


@functools.lru_cache(maxsize=256)
def _truncation_metas(svd, kept):
    """apply_mask records of U (columns), S and Vh (rows) for ``kept`` values per sector, the
    truncated sizes, and the gauge-fix independent shapes."""
    mu, ms, mv = [], [], []
    u = s = v = 0
    for t, ((_, _, slU, DU, slS, slV, DV), d) in enumerate(zip(svd, kept)):
        if d == 0:
            continue
        mu.append(((u, u + DU[0] * d), (DU[0], d), slU, DU, (t,)))
        ms.append(((s, s + d), d, slS, slS[1] - slS[0], (t,)))
        mv.append(((v, v + d * DV[1]), (d, DV[1]), slV, DV, (t,)))
        u, s, v = u + DU[0] * d, s + d, v + d * DV[1]
    return tuple(mu), tuple(ms), tuple(mv), u, s, v


@functools.lru_cache(maxsize=64)
def _transposed(eigh):
    """Records that transpose every eigenvector block, and the gauge-fix records of (U, U^T)."""
    tr = tuple((slU, (DU[1], DU[0]), slU, DU) for _, _, slU, DU, _ in eigh)
    fix = tuple((sl, D, slU, DU, slS, slU, DU) for sl, D, slU, DU, slS in eigh)
    return tr, fix


@functools.lru_cache(maxsize=1)
def _heff2():
    return Heff2Workload(load_trace('cfg2'))


# ----------------------------------------------------------------------------- inputs

def _generator(seed):
    return torch.Generator(device='cuda').manual_seed(seed)


def _normal(n, dtype, g):
    return torch.randn(n, dtype=dtype, device='cuda', generator=g)


def _orthonormal(n, k, dtype, g):
    return torch.linalg.qr(_normal((n, k), dtype, g))[0]


def _spectrum_matrix(svd, size, decades, noise, dtype, g):
    """Sectors with singular values falling over ``decades`` decades (with ``noise``: over the
    first half, the second half at the level of rounding noise), random singular vectors."""
    data = torch.empty(size, dtype=dtype, device='cuda')
    for sl, (m, n), *_ in svd:
        k = min(m, n)
        h = max(1, k // 2) if noise else k
        x = torch.arange(k, dtype=torch.float64, device='cuda')
        x = x + 0.3 * torch.rand(k, dtype=torch.float64, device='cuda', generator=g)
        d = 10.0 ** (-decades * x / h)
        if noise:
            d[h:] = 1e-18
        A = (_orthonormal(m, k, dtype, g) * d) @ _orthonormal(n, k, dtype, g).mH
        data[sl[0]:sl[1]] = A.reshape(-1)
    return data


def prepare(case, seed):
    g = _generator(seed)
    kind = case['kind']
    st = dict(case)
    if kind == 'lanczos':
        wl = _heff2()
        st['env'] = {}
        for name in ('L', 'R', 'W1', 'W2'):
            data = wl.data[name]
            st['env'][wl.keys[name]] = torch.from_numpy(data).cuda() if name[0] == 'W' else \
                _normal(data.size, torch.float64, g)
        st['v0'] = _normal(wl.data['AA'].size, torch.float64, g)
        _with_mode(case['mode'], lambda: wl.matvec(st['v0'], st['env'], backend.dot, backend.transpose_and_merge,
                                                   _scale))  # the operator's plans
        return st
    dtype = DTYPES[case['dtype']]
    grad = case.get('grad', False)
    if kind == 'tensordot':
        op, c, _ = _tensordot_structure(case['D1'], case['w1'], case['D2'], case['w2'])
        st['A'] = _normal(op.size, dtype, g).requires_grad_(grad)
        st['B'] = _normal(op.size, dtype, g).requires_grad_(grad)
        st['cot'] = _normal(c.size, dtype, g) if grad else None
    elif kind == 'fuse':
        f = _fuse_structure(case['D'], case['w'], case['order'], case['split'])
        st['A'] = _normal(f.size, dtype, g).requires_grad_(grad)
        st['cot'] = _normal(f.new_size, dtype, g) if grad else None
    elif kind == 'svd':
        ms = _matrix_structure(case['D'], case['w'], case['ratio'])
        st['A'] = _spectrum_matrix(ms['svd'], ms['size'], case['decades'], case['noise'], dtype, g)
        st['A'].requires_grad_(grad)
        if grad:
            st['cot'] = [_normal(ms['svd_sizes'][0], dtype, g), _normal(ms['svd_sizes'][1], torch.float64, g),
                         _normal(ms['svd_sizes'][2], dtype, g)]
    elif kind == 'qr':
        ms = _matrix_structure(case['D'], case['w'], case['ratio'])
        st['A'] = _normal(ms['size'], dtype, g).requires_grad_(grad)
        if grad:
            st['cot'] = [_normal(n, dtype, g) for n in ms['qr_sizes']]
    else:
        ms = _matrix_structure(case['D'], case['w'], 1.0)
        st['A'] = _normal(ms['size'], dtype, g)
        for sl, D, *_ in ms['eigh']:
            X = st['A'][sl[0]:sl[1]].view(D)
            X.copy_(X + X.mH.clone())
    return st


# ----------------------------------------------------------------------------- one pass

def run(state):
    return _RUN[state['kind']](state)


def _with_mode(mode, fn):
    before = backend.get_gemm_mode()
    backend.set_gemm_mode(mode)
    try:
        return fn()
    finally:
        backend.set_gemm_mode(before)


def _tensordot(st):
    return _with_mode(st['mode'], lambda: _tensordot_pass(st))


def _tensordot_pass(st):
    op, c, dot = _tensordot_structure(st['D1'], st['w1'], st['D2'], st['w2'])
    Am = backend.transpose_and_merge(st['A'], op.order, op.meta_new, op.meta_mrg, op.new_size)
    Bm = backend.transpose_and_merge(st['B'], op.order, op.meta_new, op.meta_mrg, op.new_size)
    C = backend.unmerge(backend.dot(Am, Bm, dot, c.new_size), c.meta_unmerge)
    if not st['grad']:
        return {'C': C}
    gA, gB = torch.autograd.grad(C, (st['A'], st['B']), st['cot'])
    return {'C': C, 'gA': gA, 'gB': gB}


def _fuse(st):
    f = _fuse_structure(st['D'], st['w'], st['order'], st['split'])
    M = backend.transpose_and_merge(st['A'], f.order, f.meta_new, f.meta_mrg, f.new_size)
    if not st['grad']:
        return {'M': M}
    return {'M': M, 'gA': torch.autograd.grad(M, st['A'], st['cot'])[0]}


def _svd(st):
    ms = _matrix_structure(st['D'], st['w'], st['ratio'])
    svd = ms['svd']
    U, S, V = backend.svd(st['A'], svd, ms['svd_sizes'])
    U, V = backend.fix_svd_signs(U, V, svd)
    slices = [rec[4] for rec in svd]
    mask, kept = ops.truncation_mask_data(S.detach(), slices, [(t,) for t in range(len(svd))], tol=TOL,
                                          D_block=_kept(st, svd), D_total=st['D'])
    mu, msd, mv, nu, ns, nv = _truncation_metas(svd, tuple(kept))
    masks = {(t,): backend.to_mask(mask[lo:hi]) for t, (lo, hi) in enumerate(slices)}
    U = backend.apply_mask(U, masks, mu, nu, 1, 2)
    S = backend.apply_mask(S, masks, msd, ns, 0, 1)
    V = backend.apply_mask(V, masks, mv, nv, 0, 2)
    out = {'U': U, 'S': S, 'V': V}
    if st['grad']:
        cot = [c[:x.numel()] for c, x in zip(st['cot'], (U, S, V))]
        out['gA'] = torch.autograd.grad((U, S, V), st['A'], cot)[0]
    return out


def _kept(case, svd):
    """Largest number of values kept per sector."""
    return max(1, int(case['keep'] * case['D'] / len(svd)))


def _qr(st):
    ms = _matrix_structure(st['D'], st['w'], st['ratio'])
    Q, R = backend.qr(st['A'], ms['qr'], ms['qr_sizes'])
    if not st['grad']:
        return {'Q': Q, 'R': R}
    return {'Q': Q, 'R': R, 'gA': torch.autograd.grad((Q, R), st['A'], st['cot'])[0]}


def _eigh(st):
    ms = _matrix_structure(st['D'], st['w'], 1.0)
    S, U = backend.eigh(st['A'], ms['eigh'], ms['eigh_sizes'])
    tr, fix = _transposed(ms['eigh'])
    U, _ = backend.fix_svd_signs(U, backend.transpose(U, (1, 0), tr), fix)  # the eigenvectors' signs made unique
    return {'S': S, 'U': U}


def _scale(x, factor):
    return x if factor == 1.0 else x * factor


def _lanczos(st):
    wl = _heff2()

    def matvec(v):
        return wl.matvec(v, st['env'], backend.dot, backend.transpose_and_merge, _scale)

    with ops.hold_constant_operands():
        res = _with_mode(st['mode'], lambda: krylov.lanczos(matvec, st['v0'], st['ncv']))
    return {'alpha': res.alpha, 'beta': res.beta, 'V': res.V}


_RUN = dict(tensordot=_tensordot, fuse=_fuse, svd=_svd, qr=_qr, eigh=_eigh, lanczos=_lanczos)


# ----------------------------------------------------------------------------- the work of a pass

def work(case):
    kind = case['kind']
    if kind == 'lanczos':
        wl, n = _heff2(), case['ncv']
        size = wl.data['AA'].size
        fixed = sum(wl.data[x].size for x in ('L', 'R', 'W1', 'W2'))
        return {'bytes': 8.0 * (fixed + size * (n + 2)), 'flops': float(n * (wl.flops + 10 * size))}
    item = {'f64': 8, 'c128': 16, 'f32': 4}[case['dtype']]
    f = 4 if case['dtype'] == 'c128' else 1
    grad = case.get('grad', False)
    if kind == 'tensordot':
        op, c, dot = _tensordot_structure(case['D1'], case['w1'], case['D2'], case['w2'])
        fl = 2 * f * sum(D[0] * D[1] * Dc[1] for _, Dc, _, D, _, _ in dot)
        return {'bytes': float(item * (2 * op.size + c.size) * (2 if grad else 1)), 'flops': float(fl * (3 if grad else 1))}
    if kind == 'fuse':
        f5 = _fuse_structure(case['D'], case['w'], case['order'], case['split'])
        return {'bytes': float(item * (f5.size + f5.new_size) * (2 if grad else 1)), 'flops': 0.0}
    ms = _matrix_structure(case['D'], case['w'], case.get('ratio', 1.0))
    shapes = [rec[1] for rec in ms['svd']]
    if kind == 'svd':    # bidiagonal reduction, both factors (14 L k^2 + 8 k^3); adjoint: 6 products
        fl = sum(14 * max(s) * min(s) ** 2 + 8 * min(s) ** 3 for s in shapes)
        fl += sum(12 * max(s) * min(s) ** 2 for s in shapes) if grad else 0
        by = item * (ms['size'] * (2 if grad else 1)) + case['keep'] * item * (ms['svd_sizes'][0] + ms['svd_sizes'][2])
    elif kind == 'qr':   # factorisation and the explicit Q; adjoint: 4 products
        fl = sum(4 * m * min(m, n) * n - 4 * min(m, n) ** 3 / 3 for m, n in shapes) * (3 if grad else 1)
        by = item * (ms['size'] + sum(ms['qr_sizes'])) * (2 if grad else 1)
    else:                # tridiagonal reduction, eigenvectors
        fl = sum(9 * n ** 3 for _, n in shapes)
        by = item * 2 * ms['size']
    return {'bytes': float(by), 'flops': float(f * fl)}


# ----------------------------------------------------------------------------- the results in 64 bits

def _merge64(data, order, meta_new, meta_mrg, size):
    out = data.new_zeros(size)
    new = {q: (D, sl) for q, D, sl in meta_new}
    for q, sl, D, sub, shape in meta_mrg:
        Dn, sn = new[q]
        block = data[sl[0]:sl[1]].view(D).permute(order).reshape(shape)
        out[sn[0]:sn[1]].view(Dn)[tuple(slice(a, b) for a, b in sub)] = block
    return out


def _merge64_adjoint(g, order, meta_new, meta_mrg, size):
    out = g.new_zeros(size)
    new = {q: (D, sl) for q, D, sl in meta_new}
    inverse = [order.index(i) for i in range(len(order))]
    for q, sl, D, sub, shape in meta_mrg:
        Dn, sn = new[q]
        block = g[sn[0]:sn[1]].view(Dn)[tuple(slice(a, b) for a, b in sub)]
        out[sl[0]:sl[1]] = block.reshape([D[i] for i in order]).permute(inverse).reshape(-1)
    return out


def _dot64(A, B, meta, size):
    out = A.new_zeros(size)
    for slc, Dc, sla, Da, slb, Db in meta:
        out[slc[0]:slc[1]] = (A[sla[0]:sla[1]].view(Da) @ B[slb[0]:slb[1]].view(Db)).reshape(-1)
    return out


def _unmerge64(data, meta):
    out = torch.empty_like(data)
    for sl, D, so, Do, sub in meta:
        out[sl[0]:sl[1]] = data[so[0]:so[1]].view(Do)[tuple(slice(a, b) for a, b in sub)].reshape(-1)
    return out


def _unmerge64_adjoint(g, meta):
    out = torch.zeros_like(g)
    for sl, D, so, Do, sub in meta:
        out[so[0]:so[1]].view(Do)[tuple(slice(a, b) for a, b in sub)] = \
            g[sl[0]:sl[1]].view([b - a for a, b in sub])
    return out


def _phases(U):
    """The phase of each column's largest entry (first row of the largest int64(|U| 2^40))."""
    rows = np.argmax((np.abs(U) * 2.0 ** 40).astype(np.int64), axis=0)
    top = U[rows, np.arange(U.shape[1])]
    return top / np.abs(top)


def exact(case, seed):
    kind = case['kind']
    st = prepare(case, seed)
    host = {k: v.detach().cpu() for k, v in st.items() if isinstance(v, torch.Tensor)}
    if case.get('dtype') == 'f32':
        host = {k: v.double() for k, v in host.items()}
    if kind == 'tensordot':
        op, c, dot = _tensordot_structure(case['D1'], case['w1'], case['D2'], case['w2'])
        A, B = (_merge64(host[x], op.order, op.meta_new, op.meta_mrg, op.new_size) for x in 'AB')
        out = {'C': _unmerge64(_dot64(A, B, dot, c.new_size), c.meta_unmerge)}
        if case['grad']:
            G = _unmerge64_adjoint(host['cot'], c.meta_unmerge)
            gA, gB = torch.zeros_like(A), torch.zeros_like(B)
            for slc, Dc, sla, Da, slb, Db in dot:
                X = G[slc[0]:slc[1]].view(Dc)
                gA[sla[0]:sla[1]] = (X @ B[slb[0]:slb[1]].view(Db).mH).reshape(-1)
                gB[slb[0]:slb[1]] = (A[sla[0]:sla[1]].view(Da).mH @ X).reshape(-1)
            out['gA'], out['gB'] = (_merge64_adjoint(x, op.order, op.meta_new, op.meta_mrg, op.size) for x in (gA, gB))
        return out
    if kind == 'fuse':
        f = _fuse_structure(case['D'], case['w'], case['order'], case['split'])
        out = {'M': _merge64(host['A'], f.order, f.meta_new, f.meta_mrg, f.new_size)}
        if case['grad']:
            out['gA'] = _merge64_adjoint(host['cot'], f.order, f.meta_new, f.meta_mrg, f.size)
        return out
    if kind == 'lanczos':
        wl = _heff2()
        env = {k: v.cpu() for k, v in st['env'].items()}
        v = host['v0']
        beta = [torch.linalg.norm(v)]
        V, alpha = [v / beta[0]], []
        for j in range(case['ncv']):
            w = wl.matvec(V[j], env, _dot64, _merge64, _scale)
            alpha.append(torch.dot(V[j], w))
            w = w - alpha[j] * V[j] - (beta[j] * V[j - 1] if j else 0)
            beta.append(torch.linalg.norm(w))
            V.append(w / beta[-1])
        return {'alpha': torch.stack(alpha), 'beta': torch.stack(beta[1:] + beta[:1]), 'V': torch.stack(V)}
    A = host['A'].numpy()
    ms = _matrix_structure(case['D'], case['w'], case.get('ratio', 1.0))
    if kind == 'qr':
        out = {'Q': [], 'R': []}
        for sl, D, *_ in ms['qr']:
            Q, R = np.linalg.qr(A[sl[0]:sl[1]].reshape(D))
            d = np.diagonal(R)
            p = d / np.abs(d)
            out['Q'].append((Q * p).reshape(-1))
            out['R'].append((R * p.conj()[:, None]).reshape(-1))
        out = {k: np.concatenate(v) for k, v in out.items()}
    elif kind == 'eigh':
        out = {'S': [], 'U': []}
        for sl, D, *_ in ms['eigh']:
            S, U = np.linalg.eigh(A[sl[0]:sl[1]].reshape(D))
            out['S'].append(S)
            out['U'].append((U / _phases(U)).reshape(-1))
        out = {k: np.concatenate(v) for k, v in out.items()}
    else:
        parts = []
        for sl, D, *_ in ms['svd']:
            U, S, V = np.linalg.svd(A[sl[0]:sl[1]].reshape(D), full_matrices=False)
            p = _phases(U)
            parts.append((U / p, S, V * p[:, None]))
        top = max(S[0] for _, S, _ in parts)
        n = [min(int(np.sum(S > TOL * top)), _kept(case, ms['svd'])) for _, S, _ in parts]
        out = {'U': np.concatenate([U[:, :d].reshape(-1) for (U, _, _), d in zip(parts, n)]),
               'S': np.concatenate([S[:d] for (_, S, _), d in zip(parts, n)]),
               'V': np.concatenate([V[:d].reshape(-1) for (_, _, V), d in zip(parts, n)])}
    if case.get('grad'):
        out['gA'] = None  # the adjoints have no plain counterpart here
    return out
