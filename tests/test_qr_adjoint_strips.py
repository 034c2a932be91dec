"""The QR adjoint's M = U gU^H - gQ^H Q in row strips (only the lower triangle is used): the strips
cover each row once, and their products, evaluated from the records, are the lower triangle of the
whole product for every height around a strip's edge, wide and tall blocks, real and complex."""
import numpy as np
import pytest

from yastn_gb300 import _plans as P


@pytest.mark.parametrize('k', list(range(1, 5)) + [31, 32, 33, 63, 64, 65, 95, 96, 97, 128, 160, 200, 432])
def test_strips_cover_the_rows(k):
    strips = P._lower_strips(k)
    assert [r for i0, i1 in strips for r in range(i0, i1)] == list(range(k))
    assert all(i1 - i0 >= 32 for i0, i1 in strips) or len(strips) == 1
    assert all(i1 - i0 < 96 for i0, i1 in strips)


def _evaluate(out_list, a, b, c, alpha):
    for off, m, n, ldc, terms in out_list:
        acc = np.zeros((m, n), dtype=c.dtype)
        for ao, bo, K, ar, ak, bk, bc, cj in terms:
            A = a[ao + ar * np.arange(m)[:, None] + ak * np.arange(K)[None, :]]
            B = b[bo + bk * np.arange(K)[:, None] + bc * np.arange(n)[None, :]]
            acc += (A.conj() if cj & 1 else A) @ (B.conj() if cj & 2 else B)
        c[off + ldc * np.arange(m)[:, None] + np.arange(n)[None, :]] += alpha * acc


@pytest.mark.parametrize('cplx', [False, True])
@pytest.mark.parametrize('m,n', [(1, 1), (40, 31), (70, 65), (64, 64), (65, 90), (130, 129), (97, 200), (160, 96)])
def test_lower_triangle_from_the_records(m, n, cplx):
    rng = np.random.default_rng(m + n)
    k = min(m, n)
    rand = lambda *s: rng.normal(size=s) + (1j * rng.normal(size=s) if cplx else 0)
    meta = (((0, m * n), (m, n), (0, m * k), (m, k), (0, k * n), (k, n)),)
    plan = P.qr_plan(meta, cplx)
    R, gR, Q, gQ = np.triu(rand(k, n)), rand(k, n), rand(m, k), rand(m, k)
    M = np.zeros(plan.m_size, dtype=R.dtype)
    _evaluate(plan.m1.out_list, R.ravel(), gR.ravel(), M, 1)
    _evaluate(plan.m2.out_list, gQ.ravel(), Q.ravel(), M, -1)
    want = R[:, :k] @ gR[:, :k].conj().T - gQ.conj().T @ Q
    # both are sums of k + m products in some order
    bound = 2 * (k + m) * 2.0 ** -52 * (np.abs(R[:, :k]) @ np.abs(gR[:, :k]).T + np.abs(gQ).T @ np.abs(Q))
    assert np.all(np.tril(np.abs(M.reshape(k, k) - want) <= 2 * bound) | ~np.tril(np.ones((k, k), bool)))
