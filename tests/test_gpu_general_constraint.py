"""The weights of the general path are distortionless: sum(w) = 1 to the roundings of w = x / sum(x) in FP32, whatever the
error of x (1 / (1^H R^-1 1) from the forward elimination leaves the sum off by that error, largest at long subarrays).
The quotient's roundings are common to the weights of a pixel, those of the weights and of the sum independent: about 2^-24
in root mean square over the pixels while ||w|| is about 1 or less (0.88 to 0.93 of it in the precise pipeline).  Bound:
1.05 of it, and 8 roundings of sum |w| at worst."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fb", [False, True])
@pytest.mark.parametrize("M,L,K", [(9, 1, 1), (16, 5, 2), (48, 24, 2), (66, 33, 1), (80, 40, 0), (126, 63, 1), (120, 56, 3)])
def test_distortionless(M, L, K, fb):
    from cos_gb300 import capon
    rng = np.random.default_rng(L)
    n, Nx = 300, 16
    Ny = n + 2 * K
    x = rng.standard_normal((Nx, Ny, M)) + 1j * rng.standard_normal((Nx, Ny, M))
    for _ in range(8):
        b0, y0 = rng.integers(Nx), rng.uniform(12, Ny - 12)
        ramp = np.exp(2j * np.pi / M * (np.arange(Nx) - b0)[:, None] * np.arange(M))
        x += 30 * np.exp(-(np.arange(Ny) - y0) ** 2 / 32)[None, :, None] * ramp[:, None, :]
    _, _, w = capon.getCaponGPU(x.astype(np.complex64), 0.01, L, K, None, fb)
    w = w.astype(np.complex128)
    off, size = np.abs(w.sum(-1) - 1), np.abs(w).sum(-1)
    assert np.all(off <= 8 * 2.0 ** -24 * size), (off / size).max() * 2 ** 24
    scale = np.maximum(1, np.linalg.norm(w, axis=-1))
    rms = np.sqrt(np.mean((off / scale) ** 2)) * 2 ** 24
    assert rms <= 1.05, rms
