"""The block SVD's sweeps where a CTA has several items (pairs of super-vectors, of up to 16 rows in FP32 and
8 in FP64 and at least one item per block): more blocks than CTAs, and blocks of so many full-rank rows
that their items alone are more than the SMs. Rows of the register kernels, tolerances of the block
SVD's other tests."""
import numpy as np
import pytest
import torch

from yastn_gb300 import ops

pytestmark = pytest.mark.gpu


def _run(blocks):
    meta, a, u, s, v = [], 0, 0, 0, 0
    for m, n in (A.shape for A in blocks):
        k = min(m, n)
        meta.append(((a, a + m * n), (m, n), (u, u + m * k), (m, k), (s, s + k), (v, v + k * n), (k, n)))
        a, u, s, v = a + m * n, u + m * k, s + k, v + k * n
    U, S, V = (x.cpu().numpy() for x in ops.svd(torch.from_numpy(np.concatenate([A.ravel() for A in blocks])).cuda(),
                                                tuple(meta), (u, s, v)))
    for A, r in zip(blocks, meta):
        Ub, Sb, Vb = U[slice(*r[2])].reshape(r[3]), S[slice(*r[4])], V[slice(*r[5])].reshape(r[6])
        k = Sb.size
        assert np.abs(Sb - np.linalg.svd(A, compute_uv=False)).max() <= 1e-12 * np.linalg.norm(A, 2)
        assert np.abs((Ub * Sb) @ Vb - A).max() <= 1e-12 * np.abs(A).max() * max(1, k)
        assert np.abs(Ub.conj().T @ Ub - np.eye(k)).max() <= 1e-12 * max(10, k)
        assert np.abs(Vb @ Vb.conj().T - np.eye(k)).max() <= 1e-12 * max(10, k)


def _draw(rng, m, n, cplx):
    return rng.normal(size=(m, n)) + (1j * rng.normal(size=(m, n)) if cplx else 0)


@pytest.mark.parametrize('cplx', [False, True])
@pytest.mark.parametrize('lo,hi', [(1, 40), (20, 70)])
def test_more_blocks_than_ctas(lo, hi, cplx, cuda_device):
    """700 blocks, wide, square and tall, some of them of low rank or zero."""
    rng = np.random.default_rng(lo + cplx)
    blocks = []
    for i in range(700):
        m, n = (int(x) for x in rng.integers(lo, hi, 2))
        A = _draw(rng, m, n, cplx)
        if i % 7 == 0:
            r = max(1, min(m, n) // 2)
            A = _draw(rng, m, r, cplx) @ _draw(rng, r, n, cplx)
        blocks.append(0 * A if i % 50 == 3 else A)
    _run(blocks)


@pytest.mark.parametrize('cplx,shapes', [(False, [(1296, 1296)] * 2), (True, [(600, 600)] * 5)])
def test_more_items_than_sms(cplx, shapes, cuda_device):
    rng = np.random.default_rng(9)
    _run([_draw(rng, m, n, cplx) for m, n in shapes])


def test_many_eigh_blocks(cuda_device):
    rng = np.random.default_rng(4)
    meta, mats, a, s = [], [], 0, 0
    for _ in range(700):
        n = int(rng.integers(1, 60))
        A = _draw(rng, n, n, True)
        mats.append(A + A.conj().T)
        meta.append(((a, a + n * n), (n, n), (a, a + n * n), (n, n), (s, s + n)))
        a, s = a + n * n, s + n
    S, U = (x.cpu().numpy() for x in ops.eigh(torch.from_numpy(np.concatenate([m.ravel() for m in mats])).cuda(),
                                              tuple(meta), (s, a)))
    for A, (_, D, slU, _, slS) in zip(mats, meta):
        w, v, n = S[slice(*slS)], U[slice(*slU)].reshape(D), D[0]
        nrm = np.linalg.norm(A, 2)
        assert np.abs(w - np.linalg.eigvalsh(A)).max() <= 1e-12 * nrm
        assert np.abs((v * w) @ v.conj().T - A).max() <= 1e-12 * nrm * max(1, n)
        assert np.abs(v.conj().T @ v - np.eye(n)).max() <= 1e-12 * max(10, n)
