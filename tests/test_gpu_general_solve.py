"""The rounding of the general path's solve stage at its longest subarrays, where it adds up: w against 64 bits, root mean
square over some hundred pixels, next to an FP32 Cholesky factorisation of the same rounded covariance.  The two make the
same roundings in another order, so the errors are equal but for chance, less than 0.05 over the pixels taken here; with
two roundings where the factorisation has one they would be up to sqrt(2) apart.  Bound: 1.1."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
f4 = np.float32


def fma(a, b, c):
    return (a.astype(np.float64) * b + c).astype(f4)


def cholesky_x(Re, Im):
    """R^-1 1 in FP32; Re, Im [n][L][L]."""
    n, L, _ = Re.shape
    A, B = Re.copy(), Im.copy()
    vr, vi = np.ones((n, L), f4), np.zeros((n, L), f4)
    iu = np.zeros((n, L), f4)
    for i in range(L):
        iu[:, i] = (1 / np.sqrt(A[:, i, i].astype(np.float64))).astype(f4)
        for v in (A, B):
            v[:, i, i + 1:] *= iu[:, i, None]
        vr[:, i] *= iu[:, i]
        vi[:, i] *= iu[:, i]
        ur, ui, yr, yi = A[:, i, i + 1:], B[:, i, i + 1:], vr[:, i, None], vi[:, i, None]
        vr[:, i + 1:] -= fma(ur, yr, ui * yi)
        vi[:, i + 1:] -= fma(ur, yi, -(ui * yr))
        kr, ki, jr, ji = ur[:, :, None], ui[:, :, None], ur[:, None, :].copy(), ui[:, None, :].copy()
        A[:, i + 1:, i + 1:] -= fma(kr, jr, ki * ji)
        B[:, i + 1:, i + 1:] -= fma(kr, ji, -(ki * jr))
    for i in range(L - 1, -1, -1):
        vr[:, i] *= iu[:, i]
        vi[:, i] *= iu[:, i]
        xr, xi, u, v = vr[:, i, None], vi[:, i, None], A[:, :i, i], B[:, :i, i]
        vr[:, :i] -= fma(u, xr, -(v * xi))
        vi[:, :i] -= fma(u, xi, v * xr)
    return vr + 1j * vi.astype(np.float64)


@pytest.mark.parametrize("L", [48, 56, 64])
def test_weights_rounding(L):
    from cos_gb300 import capon
    from test_gpu_general_exact import exact_R
    M, K, n, d = 2 * L, 1, 40, 0.01
    rng = np.random.default_rng(L)
    Ny = n + 2 * K
    x = rng.standard_normal((4, Ny, M)) + 1j * rng.standard_normal((4, Ny, M))
    for b in range(4):
        amp = (0, 0, 3, 3)[b]   # with strong signals one eigenvector dominates the error
        x[b] += amp * np.exp(-(np.arange(Ny) - Ny / 2) ** 2 / 64)[:, None] * np.exp(0.2j * (b + 1) * np.arange(M))
    x = x.astype(np.complex64)
    _, _, w = capon.getCaponGPU(x, d, L, K, None, True)
    R = exact_R(x, L, K, 1, d).reshape(-1, L, L)
    bare = exact_R(x, L, K, 1, 0).reshape(-1, L, L)
    loading = f4(d) * np.einsum("nkk->n", bare).real.astype(f4) / f4(L)
    Re, Im = bare.real.astype(f4), bare.imag.astype(f4)
    Re[:, np.arange(L), np.arange(L)] += loading[:, None]
    weights = lambda v: v / v.sum(1, keepdims=True)
    ref = weights(np.linalg.solve(R, np.ones((R.shape[0], L, 1)))[..., 0])
    rms = lambda v: np.sqrt(np.mean((np.abs(v - ref) / np.abs(ref).max(1, keepdims=True)) ** 2, axis=1))
    ratio = np.exp(np.mean(np.log(rms(w.reshape(-1, L)) / rms(weights(cholesky_x(Re, Im))))))
    assert ratio <= 1.1, ratio
