"""The 32 x 32 tiles with K chunks of the native grouped GEMM (P.fine_gemm, yb_grouped_gemm_fine):
on the CPU the records cover every output and every contracted index once; on the GPU every form
of operand at the edges of tiles, steps and chunks against NumPy, within K eps |A| |B| element by
element (the bound of any order of summation)."""
import numpy as np
import pytest

from yastn_gb300 import _plans as P

# (m, n, [K of each term])
OUTPUTS = [(31, 33, [24]), (32, 32, [25]), (33, 31, [15, 17]), (1, 40, [30]), (9, 16, [47, 1, 16]), (64, 65, [129]),
           (97, 17, [200]), (200, 3, [33]), (5, 5, [3])]


def _plan(rng, cplx, conj=True):
    lst, ao, bo, co = [], 0, 0, 0
    for i, (m, n, ks) in enumerate(OUTPUTS):
        terms = []
        for j, K in enumerate(ks):
            ta, tb = (i + j) % 2, (i + j) // 2 % 2
            fl = ((i + 2 * j) % 4) if cplx and conj else 0
            terms.append((ao, bo, K, 1 if ta else K, m if ta else 1, 1 if tb else n, K if tb else 1, fl))
            ao, bo = ao + m * K, bo + K * n
        lst.append((co, m, n, n + 2, terms))
        co += m * (n + 2)
    return P._pack_gemm(lst), lst, ao, bo, co


def test_records_cover_outputs_and_contractions():
    plan, lst, *_ = _plan(np.random.default_rng(0), False)
    f = P.fine_gemm(plan)
    assert f is not None and f is P.fine_gemm(plan)
    mine = {o[0]: o for o in lst}
    seen = {}
    for oi, tr, tc, _ in f.tiles:
        seen.setdefault(int(oi), set()).add((int(tr), int(tc)))
    got = {}
    for oi, o in enumerate(f.outs):
        m, n = int(o[1]), int(o[2])
        assert seen[oi] == {(i, j) for i in range(-(-m // 32)) for j in range(-(-n // 32))}
        if not o[6]:
            got[int(o[0])] = [tuple(int(x) for x in t) for t in f.terms[int(o[4]):int(o[5])]]
    red_of = {int(r[4]): r for r in f.red}
    for p_off, r in red_of.items():
        m, n = int(r[1]), int(r[2])
        parts = sorted((int(o[0]), int(o[4]), int(o[5])) for o in f.outs if o[6] and p_off <= o[0] < p_off + int(r[5]) * m * n)
        assert [p[0] for p in parts] == [p_off + c * m * n for c in range(int(r[5]))]
        got[int(r[0])] = [tuple(int(x) for x in t) for _, a, b in parts for t in f.terms[a:b]]
        assert sorted(int(it) for ri, it in f.tasks if f.red[ri][4] == p_off) == list(range(-(-m * n // P.GEMM_RED_ITEM)))
    rest = {int(o[0]) for o in f.rest.outs} if f.rest is not None else set()
    assert set(got) | rest == set(mine) and not set(got) & rest
    for c, terms in got.items():
        for t in mine[c][4]:  # the pieces of each term, in order, are its range
            pieces = [p for p in terms if (p[0] - t[0]) % max(t[4], 1) == 0 and p[3:] == t[3:] and
                      t[0] <= p[0] < t[0] + t[2] * max(t[4], 1) and t[1] <= p[1] < t[1] + t[2] * max(t[5], 1)]
            at = 0
            for p in pieces:
                if (p[0], p[1]) == (t[0] + at * t[4], t[1] + at * t[5]):
                    at += p[2]
            assert at == t[2]


@pytest.mark.gpu
@pytest.mark.parametrize('alpha,beta', [(1.0, 0.0), (-0.5, 1.5)])
@pytest.mark.parametrize('cplx', [False, True])
def test_kernel_at_edges(cplx, alpha, beta, cuda_device):
    import torch
    from yastn_gb300 import ops
    rng = np.random.default_rng(3)
    plan, lst, na, nb, nc = _plan(rng, cplx)

    def draw(n):
        return rng.normal(size=n) + (1j * rng.normal(size=n) if cplx else 0)
    a, b, c = draw(na), draw(nb), draw(nc)
    want, bound = c.copy(), np.zeros(nc)
    for c_off, m, n, ldc, terms in lst:
        acc, mag, kk = np.zeros((m, n), dtype=c.dtype), np.zeros((m, n)), 0
        for ao, bo, K, ars, acs, brs, bcs, fl in terms:
            A = a[ao + np.arange(m)[:, None] * ars + np.arange(K)[None, :] * acs]
            B = b[bo + np.arange(K)[:, None] * brs + np.arange(n)[None, :] * bcs]
            A, B = (A.conj() if fl & 1 else A), (B.conj() if fl & 2 else B)
            acc, mag, kk = acc + A @ B, mag + np.abs(A) @ np.abs(B), kk + K
        at = c_off + np.arange(m)[:, None] * ldc + np.arange(n)[None, :]
        want[at] = alpha * acc + beta * c[at]
        bound[at] = 4 * (kk + 3) * 2.0 ** -53 * (abs(alpha) * mag + abs(beta) * np.abs(c[at]))
    d = torch.from_numpy(c.copy()).cuda()
    ops.run_gemm(plan, torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda(), d, alpha, beta)
    assert np.all(np.abs(d.cpu().numpy() - want) <= bound)  # outside the outputs: unchanged
