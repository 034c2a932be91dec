"""Block SVD of blocks with equal singular values: the last sweep's rotations by large angles, of rows of
equal norm, leave nothing of the cosines with other rows. Tolerances of the block SVD's other tests."""
import numpy as np
import pytest
import torch

from yastn_gb300 import ops

pytestmark = pytest.mark.gpu


def _block(rng, m, n, cplx, values):
    A = rng.normal(size=(m, n)) + (1j * rng.normal(size=(m, n)) if cplx else 0)
    U, _, V = np.linalg.svd(A, full_matrices=False)
    s = rng.choice(values, size=min(m, n))
    return (U * s) @ V, np.sort(s)[::-1]


# the sweeps on registers, on super-vectors in shared memory and one pair per warp; from R's rows and A's
@pytest.mark.parametrize('qr', [True, False])
@pytest.mark.parametrize('sweeps', ['rows', 'super', 'pairs'])
@pytest.mark.parametrize('cplx', [False, True])
def test_equal_singular_values(cplx, sweeps, qr, cuda_device, monkeypatch):
    monkeypatch.setattr(ops, 'SVD_QR', [qr])
    if sweeps == 'super':
        monkeypatch.setattr(ops, 'ROWS_PER_SUPER', [4])
    elif sweeps == 'pairs':
        monkeypatch.setattr(ops, 'BLOCKED_FP64', [False])
    rng = np.random.default_rng(3 + cplx)
    shapes = [tuple(rng.integers(3, 24, size=2)) for _ in range(60)] + [(150, 150), (60, 200)]
    blocks, meta, a, u, s, v = [], [], 0, 0, 0, 0
    for m, n in shapes:
        k = min(m, n)
        values = [1.0, 0.5, 0.25] if rng.random() < 0.7 else [1.0, 1.0 - 1e-9, 0.5, 0.5 + 1e-11, 1e-3]
        blocks.append(_block(rng, m, n, cplx, values))
        meta.append(((a, a + m * n), (m, n), (u, u + m * k), (m, k), (s, s + k), (v, v + k * n), (k, n)))
        a, u, s, v = a + m * n, u + m * k, s + k, v + k * n
    data = torch.from_numpy(np.concatenate([A.ravel() for A, _ in blocks])).cuda()
    U, S, V = (x.cpu().numpy() for x in ops.svd(data, tuple(meta), (u, s, v)))
    for (A, want), r in zip(blocks, meta):
        Ub, Sb, Vb = U[slice(*r[2])].reshape(r[3]), S[slice(*r[4])], V[slice(*r[5])].reshape(r[6])
        k = Sb.size
        assert np.abs(Sb - want).max() <= 1e-12
        assert np.abs(A - (Ub * Sb) @ Vb).max() <= 1e-12 * k
        assert np.abs(Ub.conj().T @ Ub - np.eye(k)).max() <= 1e-12 * max(10, k)
        assert np.abs(Vb @ Vb.conj().T - np.eye(k)).max() <= 1e-12 * max(10, k)
