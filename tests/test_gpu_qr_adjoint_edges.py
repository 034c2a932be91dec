"""The QR adjoint's triangular solve (yb_trsm_rt) at the edges of its 32-wide tiles and 8-row
groups: B R^{-H} against NumPy. Back substitution has a residual |X R^H - B| of at most
k eps |X| |R^H| element by element."""
import ctypes

import numpy as np
import pytest
import torch

from yastn_gb300 import _native as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('cplx', [False, True])
def test_back_substitution_edges(cplx, cuda_device):
    rng = np.random.default_rng(2)
    shapes = [(1, 1), (3, 5), (8, 31), (9, 32), (7, 33), (17, 64), (20, 65), (70, 130)]
    recs, bs, rs, bo, ro = [], [], [], 0, 0
    for rows, k in shapes:
        ldb, ldr = k + 1, k + 2
        b = rng.normal(size=(rows, ldb)) + (1j * rng.normal(size=(rows, ldb)) if cplx else 0)
        r = np.triu(rng.normal(size=(k, ldr)) + (1j * rng.normal(size=(k, ldr)) if cplx else 0))
        r[np.arange(k), np.arange(k)] = 1 + rng.uniform(size=k)
        r[:, :k][~np.eye(k, dtype=bool)] *= 0.3
        recs.append((0, k, bo, rows, ldb, ro, ldr, 0))
        bs.append(b.ravel()); rs.append(r.ravel())
        bo += b.size; ro += r.size
    B, R = np.concatenate(bs), np.concatenate(rs)
    d = [torch.from_numpy(x).cuda() for x in (B, R, np.array(recs, dtype=np.int64))]
    N.call('yb_trsm_rt', d[0].data_ptr(), d[1].data_ptr(), d[2].data_ptr(), len(recs), N.YB_C128 if cplx else N.YB_F64,
           ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    got = d[0].cpu().numpy()
    for (_, k, bo, rows, ldb, ro, ldr, _) in recs:
        b, x = (a[bo:bo + rows * ldb].reshape(rows, ldb) for a in (B, got))
        r = R[ro:ro + k * ldr].reshape(k, ldr)[:, :k]
        assert np.array_equal(x[:, k:], b[:, k:])
        res = np.abs(x[:, :k] @ r.conj().T - b[:, :k])
        assert np.all(res <= 4 * (k + 2) * 2.0 ** -53 * (np.abs(x[:, :k]) @ np.abs(r.T) + np.abs(b[:, :k])))
