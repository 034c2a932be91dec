"""An emulated dot whose native sectors run on a second stream, and whose emulated part fails: the
caller's stream waits for the second one all the same, before the output's memory is given away."""
import pytest
import torch

from yastn_gb300 import ops

pytestmark = pytest.mark.gpu


def test_join_after_a_failure(cuda_device, monkeypatch):
    # one sector of K = 48 (emulated), one of K = 8 (native)
    meta = (((0, 1600), (40, 40), (0, 1920), (40, 48), (0, 1920), (48, 40)),
            ((1600, 3200), (40, 40), (1920, 2240), (40, 8), (1920, 2240), (8, 40)))
    A, B = (torch.randn(2240, dtype=torch.float64, device='cuda') for _ in range(2))
    want = ops.dot_ozaki(A, B, meta, 3200)
    waits, wait_stream = [], torch.cuda.Stream.wait_stream

    def spy(self, other):
        waits.append((self.cuda_stream, other.cuda_stream))
        return wait_stream(self, other)

    def fail(*args, **kw):
        raise RuntimeError("an allocation failed")
    main = torch.cuda.current_stream().cuda_stream
    with monkeypatch.context() as m:
        m.setattr(torch.cuda.Stream, 'wait_stream', spy)
        m.setattr(ops, '_ozaki_run', fail)
        with pytest.raises(RuntimeError, match="an allocation failed"):
            ops.dot_ozaki(A, B, meta, 3200)
    assert len(waits) == 2
    (side, first), (last, joined) = waits
    assert first == last == main and side == joined != main
    assert torch.equal(ops.dot_ozaki(A, B, meta, 3200), want)
