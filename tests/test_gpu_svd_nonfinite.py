"""Block SVD with a NaN or an Inf in one block: S and the factor from Q of that block are NaN, and the other
blocks of the call have their own, finite and right results."""
import numpy as np
import pytest
import torch

from yastn_gb300 import _plans as P, ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('emulated', [True, False])
@pytest.mark.parametrize('value', [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize('cplx', [False, True])
@pytest.mark.parametrize('shape', [(30, 30), (24, 50), (50, 24), (6, 9)])
def test_only_the_bad_block_is_lost(shape, cplx, value, emulated, cuda_device, monkeypatch):
    monkeypatch.setattr(ops, 'SVD_EMULATED', [emulated])
    rng = np.random.default_rng(shape[0] + cplx)
    shapes = [(33, 40), shape, (20, 20), (40, 33)]
    blocks = [rng.normal(size=s) + (1j * rng.normal(size=s) if cplx else 0) for s in shapes]
    blocks[1][shape[0] // 2, shape[1] // 3] = value
    meta, a, u, s, v = [], 0, 0, 0, 0
    for m, n in shapes:
        k = min(m, n)
        meta.append(((a, a + m * n), (m, n), (u, u + m * k), (m, k), (s, s + k), (v, v + k * n), (k, n)))
        a, u, s, v = a + m * n, u + m * k, s + k, v + k * n
    U, S, V = (x.cpu().numpy() for x in ops.svd(torch.from_numpy(np.concatenate([A.ravel() for A in blocks])).cuda(),
                                                tuple(meta), (u, s, v)))
    for i, (A, r) in enumerate(zip(blocks, meta)):
        Ub, Sb, Vb = U[slice(*r[2])].reshape(r[3]), S[slice(*r[4])], V[slice(*r[5])].reshape(r[6])
        if i == 1:
            if Sb.size >= P.OZAKI_MIN_DIM:
                assert np.isnan(Sb).all()
                assert np.isnan(Ub if shape[0] > shape[1] else Vb).all()
            else:  # native products: whatever they make of it, but not a finite result
                assert np.isnan(Sb).any() and np.isnan(Vb).any()
            continue
        k = Sb.size
        assert np.abs(Sb - np.linalg.svd(A, compute_uv=False)).max() <= 1e-12 * np.linalg.norm(A, 2)
        assert np.abs((Ub * Sb) @ Vb - A).max() <= 1e-12 * np.abs(A).max() * k
        assert np.abs(Ub.conj().T @ Ub - np.eye(k)).max() <= 1e-12 * k
        assert np.abs(Vb @ Vb.conj().T - np.eye(k)).max() <= 1e-12 * k


def test_an_infinite_number(cuda_device):
    """A real 1 x 1 block of infinity has it for its singular value (digits take no part in small blocks;
    a complex one is NaN in the products' own arithmetic)."""
    a = torch.full((1,), np.inf, dtype=torch.float64, device='cuda')
    U, S, V = ops.svd(a, (((0, 1), (1, 1), (0, 1), (1, 1), (0, 1), (0, 1), (1, 1)),), (1, 1, 1))
    assert S.tolist() == [np.inf]
