"""yb_svd_finalize at the sizes where its shared memory passes the 48 KB that a kernel has without
opting in (8 max_k bytes of keys; 16 max_k bytes and some static ones). The limit is sticky in a
process: each case runs in one of its own. The blocks are small, only max_k is at the edge."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = """
import sys
import torch
from yastn_gb300 import _native as N, ops, _plans as P
max_k, cplx, mode = (int(x) for x in sys.argv[1:])
dtype = torch.complex128 if cplx else torch.float64
meta = (((0, 4), (2, 2), (0, 4), (2, 2), (0, 2), (0, 4), (2, 2)),)
plan = P.svd_plan(meta, None, bool(cplx), qr=False)
r = plan.blocks[0]
work = torch.zeros(plan.n64, dtype=dtype, device='cuda')
x0, w0 = int(r[6]), int(r[7])
work[x0:x0 + 4] = torch.tensor([0., 3., 5., 0.], dtype=dtype, device='cuda')  # rows of norms 3 and 5
work[w0:w0 + 4] = torch.tensor([1., 0., 0., 1.], dtype=dtype, device='cuda')
U, V = torch.zeros(4, dtype=dtype, device='cuda'), torch.zeros(4, dtype=dtype, device='cuda')
S, shift = torch.zeros(2, dtype=torch.float64, device='cuda'), torch.ones(1, dtype=torch.float64, device='cuda')
blocks = torch.from_numpy(plan.blocks).cuda()
N.call('yb_svd_finalize', work.data_ptr(), U.data_ptr(), S.data_ptr(), V.data_ptr(), blocks.data_ptr(), 1,
       N.YB_C128 if cplx else N.YB_F64, max_k, mode, shift.data_ptr() if mode else 0, 0, 0, ops._stream())
want = [5., 3.] if mode == 0 else [2., 4.]
assert S.tolist() == want, S.tolist()
"""


@pytest.mark.parametrize('max_k,cplx,mode', [(k, c, 0) for k in (3038, 3039, 3072, 3073) for c in (0, 1)] +
                         [(2049, 0, 0), (3056, 0, 1), (8192, 1, 0)])
def test_finalize_at_shared_memory_limits(max_k, cplx, mode, cuda_device):
    res = subprocess.run([sys.executable, '-c', CHILD, str(max_k), str(cplx), str(mode)], cwd=ROOT, capture_output=True,
                         text=True, timeout=300)
    assert res.returncode == 0, res.stderr[-2000:]
