"""Block SVD of blocks scaled by powers of two: the factors do not depend on the scale and the
singular values follow it, down to norms whose squares leave FP64's range. The scaled calls differ
from the unscaled one by nothing but exponents: equal to 1e-13 (of the largest singular value)."""
import numpy as np
import pytest
import torch

from yastn_gb300 import ops

pytestmark = pytest.mark.gpu

SHAPES = [(24, 24), (20, 33), (40, 17), (5, 5), (1, 3)]


def _calls(cplx):
    """A call's blocks (eight decades of singular values), its metadata and sizes."""
    rng = np.random.default_rng(7 + cplx)
    blocks, meta, a, u, s, v = [], [], 0, 0, 0, 0
    for m, n in SHAPES:
        k = min(m, n)
        A = rng.normal(size=(m, n)) + (1j * rng.normal(size=(m, n)) if cplx else 0)
        U, _, V = np.linalg.svd(A, full_matrices=False)
        blocks.append(((U * 10.0 ** (-8 * np.arange(k) / k)) @ V).ravel())
        meta.append(((a, a + m * n), (m, n), (u, u + m * k), (m, k), (s, s + k), (v, v + k * n), (k, n)))
        a, u, s, v = a + m * n, u + m * k, s + k, v + k * n
    return np.concatenate(blocks), tuple(meta), (u, s, v)


# 2^-490: the largest rows' squares are normal, inner products and the small rows' squares are not;
# 2^-505: the squares of rows from the fourth decade on are subnormal; 2^500 the other end
@pytest.mark.parametrize('power', [-490, -505, 300, 500])
@pytest.mark.parametrize('qr,emulated', [(True, True), (True, False), (False, True)])
@pytest.mark.parametrize('cplx', [False, True])
def test_svd_of_scaled_blocks(cplx, qr, emulated, power, cuda_device):
    flat, meta, sizes = _calls(cplx)
    saved = ops.SVD_QR[0], ops.SVD_EMULATED[0]
    ops.SVD_QR[0], ops.SVD_EMULATED[0] = qr, emulated
    try:
        U0, S0, V0 = ops.svd(torch.from_numpy(flat).cuda(), meta, sizes)
        U, S, V = ops.svd(torch.from_numpy(flat * 2.0 ** power).cuda(), meta, sizes)
    finally:
        ops.SVD_QR[0], ops.SVD_EMULATED[0] = saved
    S = S.cpu().numpy() * 2.0 ** -power
    assert np.abs(S - S0.cpu().numpy()).max() <= 1e-13
    assert (U - U0).abs().max().item() <= 1e-13
    assert (V - V0).abs().max().item() <= 1e-13
