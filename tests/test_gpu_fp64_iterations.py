"""The square root, reciprocals and quotients that the sweeps, the QR and its adjoint take by iterations
in FP64 instead of CUDA's functions, over the exponent range, against NumPy in extended precision and
against sqrt and division. Bounds from the rounding errors: a step of third order from FP32's start leaves
at most 4e-20, so 1 / sqrt(u) has those of three FP64 operations (half a unit each, the first one of a term
below 1e-6): 2^-52; a chain of up to six such operations in the QR's scalars 2^-50; a quotient corrected by
its residual 2^-52."""
import ctypes

import numpy as np
import pytest

import device_functions

pytestmark = pytest.mark.gpu

LD = np.longdouble


def _run(name, *args):
    import torch
    out_like, ins = args[0], args[1:]
    d = [torch.from_numpy(np.ascontiguousarray(x)).cuda() if isinstance(x, np.ndarray) else x for x in ins]
    out = torch.zeros(out_like.shape, dtype=torch.from_numpy(out_like).dtype, device='cuda')
    n = out_like.shape[0]
    vp = [ctypes.c_void_p(x.data_ptr()) if hasattr(x, 'data_ptr') else ctypes.c_int(x) for x in d]
    st = getattr(device_functions.lib(), name)(*vp, ctypes.c_void_p(out.data_ptr()), ctypes.c_int64(n),
                                                ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert st == 0
    return out.cpu().numpy()


def _mantissas(rng, n):
    """Random significands in [1, 2), powers of two and their neighbours among them."""
    m = rng.uniform(1.0, 2.0, n)
    m[::17], m[1::17], m[2::17] = 1.0, np.nextafter(1.0, 2), np.nextafter(2.0, 1)
    return m


def test_reciprocal_square_root(cuda_device):
    u = _mantissas(np.random.default_rng(0), 200000) * np.array([1.0, 2.0, 4.0])[np.arange(200000) % 3]
    got = _run('t_rsqrt', u, u)
    assert np.abs(got.astype(LD) * np.sqrt(u.astype(LD)) - 1).max() <= LD(2) ** -52


def test_quotients(cuda_device):
    rng = np.random.default_rng(1)
    n = 300000
    v = _mantissas(rng, n) * 2.0 ** rng.integers(-500, 500, n) * rng.choice([-1.0, 1.0], n)
    d = _mantissas(rng, n) * 2.0 ** rng.integers(-480, 480, n) * rng.choice([-1.0, 1.0], n)
    got = _run('t_div', v, v, d)
    want = v.astype(LD) / d.astype(LD)
    assert np.abs((got - want) / want).max() <= LD(2) ** -52
    # zero, infinite and subnormal divisors and quotients: as the division
    v = np.array([1.0, -1.0, 0.0, 1.0, 1e300, 1e-300, 1e-310, 5e-324, np.inf, np.nan, 0.0, 1e308])
    d = np.array([0.0, 0.0, 0.0, np.inf, 1e-300, 1e300, 1e-310, 1.0, 2.0, 3.0, 7.0, 0.5])
    with np.errstate(all='ignore'):
        np.testing.assert_array_equal(_run('t_div', v, v, d), v / d)


@pytest.mark.parametrize('cplx', [False, True])
def test_reflector_scalars(cplx, cuda_device):
    rng = np.random.default_rng(2 + cplx)
    n = 300000
    e = rng.integers(-480, 480, n)

    def near():  # a value within 2^+-30 of the column's scale, now and then far below it or zero
        x = _mantissas(rng, n) * 2.0 ** (e + rng.integers(-30, 30, n)) * rng.choice([-1.0, 1.0], n)
        return np.where(rng.random(n) < 0.02, 0.0, np.where(rng.random(n) < 0.05, x * 2.0 ** -400, x))
    ar, ai = near(), near() if cplx else np.zeros(n)
    xn = _mantissas(rng, n) * 2.0 ** (2 * e)
    alpha = ar + 1j * ai if cplx else ar
    got = _run('t_scalars', np.zeros((n, 4), dtype=alpha.dtype), int(cplx), alpha, xn)
    ar, ai, xn = ar.astype(LD), ai.astype(LD), xn.astype(LD)
    sg = np.where(np.signbit(ar.astype(float)), LD(-1), LD(1))
    s = np.sqrt(ar * ar + ai * ai + xn)
    beta, d2 = -sg * s, (s + np.abs(ar)) ** 2 + ai * ai
    tau, sc, ts = 1 + np.abs(ar) / s, sg * (s + np.abs(ar)) / d2, -1 / beta
    tol = LD(2) ** -50
    parts = np.real(got)
    for c, want in ((0, tau), (1, sc), (2, beta), (3, ts)):
        assert np.abs(parts[:, c] / want - 1).max() <= tol, c
    if cplx:
        # imaginary parts to the size of the numbers
        assert (np.abs(got[:, 0].imag - ai * ts) <= tol * tau).all()
        assert (np.abs(got[:, 1].imag + ai / d2) <= tol * np.abs(sc)).all()
    # a column that is reduced already keeps its diagonal
    z = np.array([3.0, -2.0, 0.0]) + (0j if cplx else 0.0)
    got = _run('t_scalars', np.zeros((3, 4), dtype=z.dtype), int(cplx), z, np.zeros(3))
    np.testing.assert_array_equal(got, np.stack([0 * z, 0 * z, z, 0 * z], axis=1))
