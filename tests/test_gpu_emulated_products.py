"""The emulated products inside svd / eigh (P.emulated_gemm, ops.run_emulated) in every form they
take (transposed and conjugated A, transposed B, output strides, several outputs sharing an
operand, short ones on the native kernel) at tile edges, against NumPy in longdouble: the digits
hold 57 bits of each row's and column's largest element, so an entry is off by at most
K rowmax colmax 2^-55 plus one FP64 rounding of it per 400 contracted indices."""
import numpy as np
import pytest
import torch

from yastn_gb300 import _plans as P
from yastn_gb300 import ops

pytestmark = pytest.mark.gpu

FORMS = ['nn', 'tn', 'nt', 'tt']
SIZES = [(15, 15, 15), (16, 16, 16), (17, 33, 16), (63, 65, 64), (64, 64, 401), (129, 128, 127), (8, 200, 40),
         (130, 31, 900)]


@pytest.mark.parametrize('cplx', [False, True])
@pytest.mark.parametrize('form', FORMS)
def test_forms_and_edges(form, cplx, cuda_device):
    rng = np.random.default_rng(len(form) + 10 * cplx)

    def draw(m, n):
        x = rng.normal(size=(m, n)) * 10.0 ** rng.uniform(-6, 6, size=(m, 1))
        return x * np.exp(1j * rng.uniform(0, 6.28, size=(m, n))) if cplx else x
    a_parts, b_parts, lst, ref = [], [], [], []
    ao = bo = co = 0
    for m, n, K in SIZES:
        ta, tb = form[0] == 't', form[1] == 't'
        A, B = draw(*((K, m) if ta else (m, K))), draw(*((n, K) if tb else (K, n)))
        conj = int(cplx and ta)
        lst.append((co + 2, m, n, n + 3, [(ao, bo, K, 1 if ta else K, m if ta else 1, 1 if tb else n, K if tb else 1, conj)]))
        opA, opB = (A.T if ta else A), (B.T if tb else B)
        ref.append((co + 2, (opA.conj() if conj else opA), opB, n + 3))
        a_parts.append(A.ravel()); b_parts.append(B.ravel())
        ao += A.size; bo += B.size; co += m * (n + 3) + 2
    dt = torch.complex128 if cplx else torch.float64
    a, b = (torch.from_numpy(np.concatenate(x)).to(dt).cuda() for x in (a_parts, b_parts))
    c = torch.zeros(co + 8, dtype=dt, device='cuda')
    ops.run_emulated(P.emulated_gemm(lst, ops.OZAKI_SLICES, cplx), a, b, c)
    c = c.cpu().numpy()
    wide = np.clongdouble if cplx else np.longdouble
    for off, A, B, ld in ref:
        (m, K), n = A.shape, B.shape[1]
        got = np.stack([c[off + i * ld:off + i * ld + n] for i in range(m)])
        want = A.astype(wide) @ B.astype(wide)
        bound = 4 * K * np.abs(A).max(1)[:, None] * np.abs(B).max(0)[None, :] * 2.0 ** -55 * (4 if cplx else 1)
        bound = bound + 4 * (K // 400 + 2) * np.abs(want).astype(float) * 2.0 ** -53
        if K < P.OZAKI_MIN_DIM or (m <= P.OZAKI_SKINNY_ROWS and n > P.GEMM_TILE):  # native: K roundings
            bound = bound + 4 * K * (np.abs(A) @ np.abs(B)) * 2.0 ** -53
        assert np.all(np.abs((got - want).astype(complex)) <= bound)


def test_native_and_emulated_svd_agree_and_nan_propagates(cuda_device):
    rng = np.random.default_rng(5)
    n = 70
    meta = (((0, n * n), (n, n), (0, n * n), (n, n), (0, n), (0, n * n), (n, n)),)
    A = rng.normal(size=(n, n))
    data = torch.from_numpy(A.ravel()).cuda()
    S = {}
    for on in (True, False):
        saved, ops.SVD_EMULATED[0] = ops.SVD_EMULATED[0], on
        try:
            S[on] = ops.svd(data, meta, (n * n, n, n * n))[1].cpu().numpy()
        finally:
            ops.SVD_EMULATED[0] = saved
    ref = np.linalg.svd(A, compute_uv=False)
    err = {on: np.abs(s - ref).max() / ref[0] for on, s in S.items()}
    assert err[True] <= 1e-14 and err[False] <= 1e-14
    bad = data.clone()
    bad[17] = float('nan')
    out = {}
    for on in (True, False):
        saved, ops.SVD_EMULATED[0] = ops.SVD_EMULATED[0], on
        try:
            out[on] = [torch.isnan(x).any().item() for x in ops.svd(bad, meta, (n * n, n, n * n))]
        except Exception as e:  # both refuse, or both return the same kind of result
            out[on] = type(e)
        finally:
            ops.SVD_EMULATED[0] = saved
    assert out[True] == out[False]


@pytest.mark.parametrize('graded', ['rows', 'cols', 'both'])
def test_graded_matrices_keep_their_relative_accuracy(graded, cuda_device):
    """A = D B, B D or D B D over 12 decades: the emulated product X = W R is as accurate as the
    native one, singular value by singular value and (rows) row by row of U S Vh - A. The native
    path's own errors set the scale: k eps = 1e-14 relative to each value, and to each row."""
    rng = np.random.default_rng(8)
    k = 100
    d = 10.0 ** (-12 * np.arange(k) / k)
    B = rng.normal(size=(k, k))
    A = B * {'rows': d[:, None], 'cols': d[None, :], 'both': d[:, None] * d[None, :]}[graded]
    meta = (((0, k * k), (k, k), (0, k * k), (k, k), (0, k), (0, k * k), (k, k)),)
    x = torch.from_numpy(A.ravel().copy()).cuda()
    res = {}
    for on in (True, False):
        saved, ops.SVD_EMULATED[0] = ops.SVD_EMULATED[0], on
        try:
            res[on] = [t.cpu().numpy() for t in ops.svd(x, meta, (k * k, k, k * k))]
        finally:
            ops.SVD_EMULATED[0] = saved
    S = res[False][1]
    assert np.abs(res[True][1] / S - 1).max() <= 1e-13
    row = {}
    for on, (U, S, V) in res.items():
        r = (U.reshape(k, k) * S) @ V.reshape(k, k) - A
        row[on] = (np.abs(r).max(1) / np.abs(A).max(1)).max()
    assert row[True] <= max(2 * row[False], 1e-13)
