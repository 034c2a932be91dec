"""Block SVD of blocks of very low rank: nearly all vectors are completed on the host's side of the
call, and the projection onto the few others is a product of few rows and long K, which runs in K
chunks alone. Tolerances of the block SVD's other tests."""
import numpy as np
import pytest
import torch

from yastn_gb300 import _plans as P, ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('emulated', [True, False])
@pytest.mark.parametrize('cplx', [False, True])
@pytest.mark.parametrize('m,n,rank', [(300, 300, 5), (280, 400, 8), (420, 270, 1), (300, 300, 9)])
def test_completion_of_low_rank_blocks(m, n, rank, cplx, emulated, cuda_device):
    rng = np.random.default_rng(m + rank + cplx)

    def draw(*shape):
        return rng.normal(size=shape) + (1j * rng.normal(size=shape) if cplx else 0)
    A, k = draw(m, rank) @ draw(rank, n), min(m, n)
    meta = (((0, m * n), (m, n), (0, m * k), (m, k), (0, k), (0, k * n), (k, n)),)
    (cp,) = P.completion_plans(P.svd_plan(meta, None, cplx, qr=True).blocks, [k - rank], cplx)
    assert cp.e1.n_tiles or cp.e1.native.split is not None or cp.e1.native.outs.size
    saved, ops.SVD_EMULATED[0] = ops.SVD_EMULATED[0], emulated
    try:
        U, S, V = (x.cpu().numpy() for x in ops.svd(torch.from_numpy(A.ravel()).cuda(), meta, (m * k, k, k * n)))
    finally:
        ops.SVD_EMULATED[0] = saved
    U, V = U.reshape(m, k), V.reshape(k, n)
    assert np.abs(S - np.linalg.svd(A, compute_uv=False)).max() <= 1e-12 * np.linalg.norm(A, 2)
    assert np.abs((U * S) @ V - A).max() <= 1e-12 * np.abs(A).max() * k
    assert np.abs(U.conj().T @ U - np.eye(k)).max() <= 1e-12 * k
    assert np.abs(V @ V.conj().T - np.eye(k)).max() <= 1e-12 * k


def test_completion_plans_are_bounded(cuda_device):
    """The counts of completed vectors differ from call to call: the plan of the blocks does not collect
    a completion plan for each."""
    rng = np.random.default_rng(0)
    n = 260
    meta = (((0, n * n), (n, n), (0, n * n), (n, n), (0, n), (0, n * n), (n, n)),)
    for rank in range(1, 2 * ops.MAX_COMPLETIONS + 1):
        A = rng.normal(size=(n, rank)) @ rng.normal(size=(rank, n))
        ops.svd(torch.from_numpy(A.ravel()).cuda(), meta, (n * n, n, n * n))
    kept = P.svd_plan(meta, None, False, qr=True)._completion
    assert 0 < len(kept) <= ops.MAX_COMPLETIONS
