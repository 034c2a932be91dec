"""Panels factored by a cluster of two CTAs (csrc/yb_qr.cuh): the row passes of 512, columns at the
length from which a panel is shared, long and short blocks in one call, and the block counts around
which the clusters' groups change. A = Q R with a positive diagonal; the bounds are those of backward
stability with an order of magnitude to spare (1e-13 max(1, sqrt(k)))."""
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


@pytest.mark.parametrize('cplx', [False, True])
@pytest.mark.parametrize('shapes', [[(256, 70)], [(257, 70)], [(512, 21), (513, 22)], [(1024, 9), (1025, 10)],
                                    [(1536, 13), (1537, 11)], [(3072, 9)], [(3073, 9)], [(600, 600), (40, 30), (290, 310)],
                                    [(261, 33)] * 13, [(258, 9)] * 19, [(259, 9)] * 20])
def test_shared_panels(shapes, cplx, cuda_device):
    rng = np.random.default_rng(len(shapes) + shapes[0][0])
    mats = [rng.normal(size=s) + (1j * rng.normal(size=s) if cplx else 0) for s in shapes]
    mats[0][:, 3] = mats[0][:, 1]  # a dependent column
    for A, (Q, R) in zip(mats, _run(mats)):
        k = min(A.shape)
        tol = 1e-13 * max(1.0, np.sqrt(k))
        norm = np.linalg.norm(A, 2)
        assert np.linalg.norm(Q @ R - A, 2) <= tol * norm
        assert np.linalg.norm(Q.conj().T @ Q - np.eye(k), 2) <= tol
        assert np.abs(np.tril(R[:, :k], -1)).max(initial=0.0) == 0.0
        d = np.diagonal(R)
        assert np.all(d.real >= 0) and np.abs(d.imag).max() <= tol * norm
