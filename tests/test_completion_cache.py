"""The completion plans kept with a plan of the block SVD, from several threads at once: no thread's
insertion disturbs another's eviction, and the last few are kept."""
import sys
import threading
from types import SimpleNamespace

import torch

from yastn_gb300 import _plans as P, ops


def test_threads_share_the_completion_plans(monkeypatch):
    monkeypatch.setattr(P, 'completion_plans', lambda blocks, nz, cplx: [])
    monkeypatch.setattr(ops, '_stream', lambda: 0)
    plan, factor, errors = SimpleNamespace(blocks=()), torch.zeros(1), []

    def work(t):
        try:
            for i in range(5000):
                ops._complete(plan, factor, factor, (t, i), False)
        except Exception as e:
            errors.append(e)
    before = sys.getswitchinterval()
    sys.setswitchinterval(1e-6)
    try:
        threads = [threading.Thread(target=work, args=(t,)) for t in range(4)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    finally:
        sys.setswitchinterval(before)
    assert not errors
    assert 0 < len(plan._completion) <= ops.MAX_COMPLETIONS
