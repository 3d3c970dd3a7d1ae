"""Beamspace pixels without a Cholesky factor: outputs that are not finite, whatever kernel serves the beam count.

A negative absolute loading larger than R_bs makes every pivot negative.  R - |d| I with |d| just above the
smallest eigenvalue has as many negative pivots as negative eigenvalues (Sylvester's inertia): one or a few.  In both the frame's other beam, under enough signal to stay definite, keeps its values."""
import numpy as np
import pytest

from test_gpu_beamspace_rows import absolute

pytestmark = pytest.mark.gpu


def noise(rng, *shape):
    return (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).astype(np.complex64)


@pytest.mark.parametrize("indefinite", [False, True])
@pytest.mark.parametrize("Nb", [3, 5, 6, 7, 8, 9, 16, 17, 31])
def test_no_factor_is_not_finite(Nb, indefinite):
    from cos_gb300 import _lib, capon
    M, L, K, Ny = 64, 32, 1, 37
    x = noise(np.random.default_rng(Nb), 2, Ny, M)
    n, T, Ns = Ny - 2 * K, 2 * K + 1, M - L + 1
    # eigenvalues of B R B^H of the beam that is to fail, pixel by pixel
    b = np.arange(Nb)
    bins = np.where(b > Nb // 2, b + (L - 2 * (Nb // 2) - 1), b)
    B = np.exp(-2j * np.pi * np.outer(bins, np.arange(L)) / L) / np.sqrt(L)
    ev = []
    for p in range(n):
        y = np.lib.stride_tricks.sliding_window_view(x[0, p:p + T], L, axis=1).reshape(-1, L) @ B.T
        ev.append(np.linalg.eigvalsh(y.T @ y.conj() / (Ns * T)))
    ev = np.array(ev)
    d = -1.1 * ev[:, 0].max() if indefinite else -2.0 * ev[:, -1].max()
    assert (ev[:, 0] + d < -0.01).all()
    x[1] *= np.sqrt(100.0 * -d / ev[:, 0].min())
    z, P, w = capon.getCaponGPU(x, d, L, K, np.zeros((Nb, L)), loading=_lib.LOAD_ABSOLUTE)
    for v in (z[0], P[0], w[0]):
        assert not np.isfinite(v).any()
    ref = absolute(x[1:], d, L, K, Nb)
    assert np.abs(P[1] / ref["P"][0] - 1).max() <= 1e-4
    assert np.abs(w[1] - ref["w"][0]).max() <= 2e-3 * np.abs(ref["w"][0]).max()


@pytest.mark.parametrize("Nb", [5, 8, 16, 24])
def test_no_samples_is_not_finite(Nb):
    """R = 0 without loading: a zero pivot."""
    from cos_gb300 import capon
    z, P, w = capon.getCaponGPU(np.zeros((1, 20, 48), np.complex64), 0.0, 24, 1, np.zeros((Nb, 24)))
    for v in (z, P, w):
        assert not np.isfinite(v).any()
