"""The block SVD / eigh sweeps (csrc/yb_jacobi.cu) at the edges of their row lengths and
super-vectors, against LAPACK in FP64: singular values and eigenvalues within 1e-12 of the
largest, reconstruction within 1e-12 |A| max(1, k), factors orthonormal within 1e-12 max(10, k)
(the tolerances of the block SVD's other tests). Each call holds a full-rank block, a graded
rank-deficient one (half of its rows at rounding noise) and a small one."""
import numpy as np
import pytest
import torch

from yastn_gb300 import ops

pytestmark = pytest.mark.gpu


def _block(m, n, rng, cplx, rank=None):
    A = rng.normal(size=(m, n)) + (1j * rng.normal(size=(m, n)) if cplx else 0)
    if rank is None:
        return A
    U, _, V = np.linalg.svd(A, full_matrices=False)
    return (U[:, :rank] * 10.0 ** (-8 * np.arange(rank) / max(rank, 1))) @ V[:rank]


def _svd_meta(shapes):
    meta, a, u, s, v = [], 0, 0, 0, 0
    for m, n in shapes:
        k = min(m, n)
        meta.append(((a, a + m * n), (m, n), (u, u + m * k), (m, k), (s, s + k), (v, v + k * n), (k, n)))
        a, u, s, v = a + m * n, u + m * k, s + k, v + k * n
    return tuple(meta), (u, s, v)


def _check(A, U, S, V):
    k = S.size
    assert np.abs(S - np.linalg.svd(A, compute_uv=False)).max() <= 1e-12 * np.linalg.norm(A, 2)
    assert np.abs((U * S) @ V - A).max() <= 1e-12 * np.abs(A).max() * max(1, k)
    assert np.abs(U.conj().T @ U - np.eye(k)).max() <= 1e-12 * max(10, k)
    assert np.abs(V @ V.conj().T - np.eye(k)).max() <= 1e-12 * max(10, k)


REAL = [1, 2, 4, 5, 8, 9, 15, 16, 17, 31, 32, 33, 63, 64, 65, 127, 128, 129, 448, 449]
CPLX = [1, 2, 5, 16, 17, 33, 128, 129]


@pytest.mark.parametrize('k,cplx', [(k, False) for k in REAL] + [(k, True) for k in CPLX])
def test_svd_at_row_edges(k, cplx, cuda_device):
    rng = np.random.default_rng(100 * k + cplx)
    shapes = [(k, k), (k + k // 3, k), (min(k, 3), 7)]
    blocks = [_block(*shapes[0], rng, cplx), _block(*shapes[1], rng, cplx, max(1, k // 2)), _block(*shapes[2], rng, cplx)]
    meta, sizes = _svd_meta(shapes)
    data = torch.from_numpy(np.concatenate([b.ravel() for b in blocks])).cuda()
    U, S, V = (x.cpu().numpy() for x in ops.svd(data, meta, sizes))
    for A, (_, _, slU, DU, slS, slV, DV) in zip(blocks, meta):
        _check(A, U[slice(*slU)].reshape(DU), S[slice(*slS)], V[slice(*slV)].reshape(DV))


@pytest.mark.parametrize('k,cplx', [(k, False) for k in (1, 3, 4, 17, 33, 129)] + [(k, True) for k in (2, 17, 65)])
def test_eigh_at_row_edges(k, cplx, cuda_device):
    rng = np.random.default_rng(200 * k + cplx)
    meta, mats, a, s = [], [], 0, 0
    for n in (k, max(1, k // 2), 2):
        A = _block(n, n, rng, cplx)
        mats.append(A + A.conj().T)
        meta.append(((a, a + n * n), (n, n), (a, a + n * n), (n, n), (s, s + n)))
        a, s = a + n * n, s + n
    data = torch.from_numpy(np.concatenate([m.ravel() for m in mats])).cuda()
    S, U = (x.cpu().numpy() for x in ops.eigh(data, tuple(meta), (s, a)))
    for A, (_, D, slU, _, slS) in zip(mats, meta):
        w, v, n = S[slice(*slS)], U[slice(*slU)].reshape(D), D[0]
        nrm = np.linalg.norm(A, 2)
        assert np.abs(w - np.linalg.eigvalsh(A)).max() <= 1e-12 * nrm
        assert np.abs((v * w) @ v.conj().T - A).max() <= 1e-12 * nrm * max(1, n)
        assert np.abs(v.conj().T @ v - np.eye(n)).max() <= 1e-12 * max(10, n)


@pytest.mark.parametrize('k', [896, 897, 1312, 1313])
def test_singular_values_at_long_rows(k, cuda_device):
    """The longest rows of each register variant, and the first ones of the shared-memory path."""
    rng = np.random.default_rng(k)
    A = _block(k, k, rng, False, k // 2)
    meta, sizes = _svd_meta([(k, k)])
    U, S, V = (x.cpu().numpy() for x in ops.svd(torch.from_numpy(A.ravel().copy()).cuda(), meta, sizes))
    _check(A, U.reshape(k, k), S, V.reshape(k, k))
