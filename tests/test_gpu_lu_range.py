"""The batched LU solve of very small and very large systems.  The solution of s A x = s b does not depend on s, and the
solver's arithmetic leaves only the squared modulus of a pivot p near the ends of the FP32 range: below |p| = 1.1e-19 it
is subnormal, with an absolute error of half of 2^-149.  Bound: Gaussian elimination's 4 N eps cond(A), and the relative
error of that squared modulus, met in the multipliers and in the back substitution, 2 N times."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1e-20, 3e-20, 1e-19, 1e-10, 1e10, 3e18])
@pytest.mark.parametrize("N", [3, 8, 16, 24, 32, 36, 48, 72])
def test_lu_scaled(N, scale):
    from cos_gb300 import capon
    rng = np.random.default_rng(N)
    batch = 9
    noise = lambda *s: rng.standard_normal(s) + 1j * rng.standard_normal(s)
    # every pivot close to 4: the diagonal outweighs its row
    A = (scale * (4 * np.eye(N) + 0.2 / np.sqrt(N) * noise(batch, N, N))).astype(np.complex64)
    b = (scale * noise(batch, N)).astype(np.complex64)
    x = np.zeros((batch, N), np.complex64)
    assert capon.Solver().solve(x, np.ascontiguousarray(np.transpose(A, (0, 2, 1))), b, N, batch) == 0
    A64, b64 = A.astype(np.complex128) / scale, b.astype(np.complex128) / scale
    ref = np.linalg.solve(A64, b64[..., None])[..., 0]
    err = np.linalg.norm(x - ref, axis=1) / np.linalg.norm(ref, axis=1)
    pivot = scale * 3.0
    sub = 2.0 ** -150 / pivot ** 2 if pivot ** 2 < 2.0 ** -126 else 0.0
    bound = (4 * N * 2.0 ** -23 + 2 * N * sub) * np.linalg.cond(A64)
    assert np.all(err <= bound), (err / bound).max()
