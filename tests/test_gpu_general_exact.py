"""The covariance of the general element-space path is the float-float sum of exact products, rounded once: every
off-diagonal component of R within half an ulp of the FP64 one, the diagonal within two roundings (the loading is added
in FP32).  The float-float sums leave less than 2^-40 of the largest entry: 2^-47 of it for each of their at most
2 T (Ns + 2 L) < 2^13 steps would be that in the worst case, and their errors have either sign."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def exact_R(x, L, K, fb, d):
    """Unnormalised, loaded, [b][n][L][L], (row, column)."""
    x = x.astype(np.complex128)
    Nx, Ny, M = x.shape
    n, T = Ny - 2 * K, 2 * K + 1
    sub = np.lib.stride_tricks.sliding_window_view(x, L, axis=2)            # b, y, s, l
    rows = np.einsum("bysk,bysl->bykl", sub, sub.conj())
    R = sum(rows[:, t:t + n] for t in range(T))
    if fb:
        R = 0.5 * (R + np.swapaxes(R, 2, 3)[:, :, ::-1, ::-1])
    tr = np.einsum("bnkk->bn", R).real
    return R + (np.float32(d) * tr / L)[..., None, None] * np.eye(L)


# Nx, pixels, M, L, K
CASES = [(2, 9, 5, 1, 1), (2, 5, 7, 2, 0), (2, 70, 17, 8, 1), (2, 13, 33, 17, 2), (3, 40, 48, 24, 3), (2, 11, 62, 31, 4),
         (1, 6, 72, 24, 12), (1, 9, 24, 12, 60), (1, 7, 80, 40, 2), (1, 5, 126, 63, 1), (1, 4, 300, 20, 2), (1, 3, 63, 63, 2),
         (30, 150, 48, 24, 2), (1, 8, 126, 63, 16)]


@pytest.mark.parametrize("fb", [0, 1])
@pytest.mark.parametrize("Nx,n,M,L,K", CASES)
def test_rounded_once(Nx, n, M, L, K, fb):
    from cos_gb300 import capon
    rng = np.random.default_rng(M + K)
    Ny, d = n + 2 * K, 0.01
    x = rng.standard_normal((Nx, Ny, M)) + 1j * rng.standard_normal((Nx, Ny, M))
    x += 10 * np.exp(-(np.arange(Ny) - Ny / 2) ** 2 / 32)[None, :, None] * np.exp(0.3j * np.arange(M))
    x = x.astype(np.complex64)
    z, P, R = np.zeros((Nx, n), np.complex64), np.zeros((Nx, n), np.float32), np.zeros((Nx, n, L, L), np.complex64)
    assert capon.Capon().getCaponEx(z, P, None, R, x, d, L, K, M, Nx, Ny, 0, capon.opts(fb=fb)) == 0
    got, want = np.swapaxes(R, 2, 3), exact_R(x, L, K, fb, d)               # memory holds the columns
    tiny = 2.0 ** -40 * np.abs(want).max(axis=(2, 3), keepdims=True)
    rounds = 1 + np.eye(L)
    for part in (np.real, np.imag):
        err, size = np.abs(part(got).astype(np.float64) - part(want)), np.abs(part(want))
        assert np.all(err <= 2.0 ** -24 * rounds * size + tiny), (err / (2.0 ** -24 * size + tiny)).max()
