"""Block SVD of blocks graded by columns (tall ones by rows): every column of A - U S V is small against
that column of A, as an FP64 product of the factors gives it, although most columns are small against
A. Blocks that are not graded, whatever their spectrum, keep the emulated products."""
import numpy as np
import pytest
import torch

from yastn_gb300 import ops

pytestmark = pytest.mark.gpu


def _draw(rng, m, n, cplx):
    return rng.normal(size=(m, n)) + (1j * rng.normal(size=(m, n)) if cplx else 0)


def _graded(rng, m, n, decades, cplx, shuffled):
    """A generic block with its longer side's rows or columns scaled over the decades."""
    d = 10.0 ** (-decades * np.arange(max(m, n)) / max(m, n))
    if shuffled:
        d = rng.permutation(d)
    A = _draw(rng, m, n, cplx)
    return d[:, None] * A if m > n else A * d


def _spectrum(rng, m, n, decades, cplx, rank=None):
    U, _, V = np.linalg.svd(_draw(rng, m, n, cplx), full_matrices=False)
    k = min(m, n)
    r = k if rank is None else rank
    return (U[:, :r] * 10.0 ** (-decades * np.arange(r) / r)) @ V[:r]


def _svd(blocks, monkeypatch):
    meta, a, u, s, v = [], 0, 0, 0, 0
    for m, n in (A.shape for A in blocks):
        k = min(m, n)
        meta.append(((a, a + m * n), (m, n), (u, u + m * k), (m, k), (s, s + k), (v, v + k * n), (k, n)))
        a, u, s, v = a + m * n, u + m * k, s + k, v + k * n
    seen, run = [], ops._run_flagged

    def spy(guard, name, x, y, z, flags):
        seen.append(flags)
        return run(guard, name, x, y, z, flags)
    monkeypatch.setattr(ops, '_run_flagged', spy)
    U, S, V = (x.cpu().numpy() for x in ops.svd(torch.from_numpy(np.concatenate([A.ravel() for A in blocks])).cuda(),
                                                tuple(meta), (u, s, v)))
    out = [(U[slice(*r[2])].reshape(r[3]), S[slice(*r[4])], V[slice(*r[5])].reshape(r[6])) for r in meta]
    return out, seen[-1].cpu().numpy() if seen else None


# Columns in the order of their scales: shuffled, an FP64 SVD from an unpivoted QR has no such bound. Nor
# has it where a singular value is noise (at most 1e-14 of the block's norm, as the smallest one of the
# real 96 x 96 block over 12 decades): there the native products are the measure.
@pytest.mark.parametrize('decades', [6, 12])
@pytest.mark.parametrize('cplx', [False, True])
def test_columns_of_graded_blocks(cplx, decades, cuda_device, monkeypatch):
    rng = np.random.default_rng(decades + cplx)
    blocks = [_graded(rng, m, n, decades, cplx, False) for m, n in ((24, 24), (24, 36), (33, 17), (96, 96), (150, 130))]
    blocks += [_spectrum(rng, 64, 64, 8, cplx), _draw(rng, 10, 12, cplx)]
    out, flags = _svd(blocks, monkeypatch)
    with monkeypatch.context() as native:
        native.setattr(ops, 'SVD_EMULATED', [False])
        ref, _ = _svd(blocks, native)

    def left(A, U, S, V):
        axis = 1 if A.shape[0] > A.shape[1] else 0
        return np.linalg.norm(A - (U * S) @ V, axis=axis) / np.linalg.norm(A, axis=axis)
    for A, (U, S, V), r in zip(blocks, out, ref):
        assert np.all(left(A, U, S, V) <= (1e-12 if S[-1] > 1e-14 * np.linalg.norm(A) else 1e-12 + 2 * left(A, *r)))
        k = S.size
        assert np.abs(U.conj().T @ U - np.eye(k)).max() <= 1e-12 * max(10, k)
        assert np.abs(V @ V.conj().T - np.eye(k)).max() <= 1e-12 * max(10, k)
    assert flags[3] and flags[4] and not flags[5] and not flags[6]


@pytest.mark.parametrize('cplx', [False, True])
def test_spectra_alone_are_not_graded(cplx, cuda_device, monkeypatch):
    """Spectra over up to 14 decades between generic factors, and ranks with a tail of noise."""
    rng = np.random.default_rng(11 + cplx)
    blocks = [_draw(rng, 40, 40, cplx), _spectrum(rng, 100, 100, 4, cplx), _spectrum(rng, 140, 90, 9, cplx),
              _spectrum(rng, 90, 200, 9, cplx, 45), _spectrum(rng, 216, 216, 14, cplx), _spectrum(rng, 300, 300, 9, cplx, 150)]
    _, flags = _svd(blocks, monkeypatch)
    assert not flags.any(), flags
