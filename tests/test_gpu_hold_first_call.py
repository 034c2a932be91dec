"""The first emulated dot of a metadata tuple inside ``hold_constant_operands``: its kernels are
timed there, and a dot with both operands held reuses their digit planes."""
import pytest
import torch

from yastn_gb300 import ops

pytestmark = pytest.mark.gpu


def test_first_dot_inside_the_scope(cuda_device):
    m, k, n = 37, 48, 53  # sizes of this test alone: their plan is built here
    meta = (((0, m * n), (m, n), (0, m * k), (m, k), (0, k * n), (k, n)),)
    A = torch.randn(m * k, dtype=torch.float64, device='cuda')
    B = torch.randn(k * n, dtype=torch.float64, device='cuda')
    want = (A.view(m, k) @ B.view(k, n)).reshape(-1)
    with ops.hold_constant_operands():
        first = ops.dot_ozaki(A, B, meta, m * n)
        again = ops.dot_ozaki(A, B, meta, m * n)      # both operands held
        C = B * 2
        other = ops.dot_ozaki(A, C, meta, m * n)      # one held
    assert torch.allclose(first, want, rtol=0, atol=1e-12 * k)
    assert torch.equal(first, again)
    assert torch.equal(other, 2 * first)
