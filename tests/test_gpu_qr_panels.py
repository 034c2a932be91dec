"""The blocked Householder QR (csrc/yb_qr.cuh) at the edges of its panels and of the rows a panel
takes in registers: A = Q R with a positive diagonal, against LAPACK's factors made unique the
same way. Backward stability gives |A - Q R| and |Q^H Q - 1| of a few eps sqrt(k) |A|; 1e-13 |A|
max(1, sqrt(k)) bounds them with an order of magnitude to spare. Rank-deficient and zero columns
keep both (their R rows are not unique, so they are not compared)."""
import numpy as np
import pytest
import torch

from yastn_gb300 import ops

pytestmark = pytest.mark.gpu


def _run(mats):
    meta, a, q, r = [], 0, 0, 0
    for A in mats:
        m, n = A.shape
        k = min(m, n)
        meta.append(((a, a + m * n), (m, n), (q, q + m * k), (m, k), (r, r + k * n), (k, n)))
        a, q, r = a + m * n, q + m * k, r + k * n
    data = torch.from_numpy(np.concatenate([A.ravel() for A in mats])).cuda()
    Q, R = (x.cpu().numpy() for x in ops.qr(data, tuple(meta), (q, r)))
    return [(Q[slice(*m[2])].reshape(m[3]), R[slice(*m[4])].reshape(m[5])) for m in meta]


def _check(A, Q, R, unique):
    k = min(A.shape)
    tol = 1e-13 * max(1.0, np.sqrt(k))
    scale = max(np.linalg.norm(A, 2), 1e-300)
    assert np.linalg.norm(Q @ R - A, 2) <= tol * scale
    assert np.linalg.norm(Q.conj().T @ Q - np.eye(k), 2) <= tol
    assert np.abs(np.tril(R[:, :k], -1)).max(initial=0.0) == 0.0
    d = np.diagonal(R)
    assert np.all(d.real >= 0) and np.abs(d.imag).max() <= tol * scale
    if unique:
        Qr, Rr = np.linalg.qr(A)
        p = np.diagonal(Rr) / np.abs(np.diagonal(Rr))
        cond = np.linalg.cond(A[:, :k])
        assert np.abs(R - p.conj()[:, None] * Rr).max() <= tol * scale * max(cond, 1.0)


def _rand(m, n, rng, cplx):
    return rng.normal(size=(m, n)) + (1j * rng.normal(size=(m, n)) if cplx else 0)


SHAPES = [(1, 1), (1, 7), (2, 2), (3, 3), (4, 4), (5, 5), (7, 4), (8, 9), (33, 17), (64, 64), (130, 97)]


@pytest.mark.parametrize('cplx', [False, True])
def test_small_shapes_in_one_call(cplx, cuda_device):
    rng = np.random.default_rng(1)
    mats = [_rand(m, n, rng, cplx) for m, n in SHAPES]
    deficient = _rand(40, 6, rng, cplx) @ _rand(6, 30, rng, cplx)
    zero = np.zeros((12, 9), dtype=mats[0].dtype)
    holes = _rand(20, 14, rng, cplx)
    holes[:, [0, 5, 13]] = 0
    out = _run(mats + [deficient, zero, holes])
    for i, (A, (Q, R)) in enumerate(zip(mats + [deficient, zero, holes], out)):
        _check(A, Q, R, i < len(mats))


@pytest.mark.parametrize('m,n,cplx', [(511, 13, False), (512, 13, False), (513, 13, False), (1025, 10, False),
                                      (1537, 10, False), (2816, 9, False), (2817, 9, False), (2900, 21, False),
                                      (6500, 9, False), (1025, 6, True), (2820, 9, True), (3300, 9, True)])
def test_long_columns(m, n, cplx, cuda_device):
    """The row passes of a panel in registers, columns beyond them, and panels whose V does not fit
    in shared memory."""
    rng = np.random.default_rng(m + n)
    A = _rand(m, n, rng, cplx)
    (Q, R), = _run([A])
    _check(A, Q, R, True)


def test_more_blocks_than_sms(cuda_device):
    rng = np.random.default_rng(3)
    mats = [_rand(int(rng.integers(1, 40)), int(rng.integers(1, 40)), rng, False) for _ in range(400)]
    mats.append(_rand(1100, 11, rng, False))
    for A, (Q, R) in zip(mats, _run(mats)):
        _check(A, Q, R, False)
