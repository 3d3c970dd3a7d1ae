"""The batched LU solve at both sides of every register size (8, 16, 24, 32, 48, 64, 72 columns), for systems that
need their row exchanges (small leading entries), ties and a zero leading entry, against numpy in FP64.  The bound is
the one for Gaussian elimination with partial pivoting, a small multiple of N eps cond(A)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [1, 2, 7, 8, 9, 15, 16, 17, 24, 25, 31, 32, 33, 36, 37, 40, 41, 47, 48, 49, 63, 64, 65, 71, 72])
def test_lu_sizes(N):
    from cos_gb300 import capon
    rng = np.random.default_rng(N)
    batch = 37                       # a partial last block at every group size
    A = rng.standard_normal((batch, N, N)) + 1j * rng.standard_normal((batch, N, N))
    A[::3, 0, 0] *= 1e-6             # the first pivot lies below
    if N > 1:
        A[1::3, 0, 0] = 0.0
        A[2::3, :, 0] = A[2::3, :1, 0]   # equal moduli down the first column
    A = A.astype(np.complex64)
    b = (rng.standard_normal((batch, N)) + 1j * rng.standard_normal((batch, N))).astype(np.complex64)
    x = np.zeros((batch, N), np.complex64)
    Acm = np.ascontiguousarray(np.transpose(A, (0, 2, 1)))
    assert capon.Solver().solve(x, Acm, b, N, batch) == 0
    A64, b64 = A.astype(np.complex128), b.astype(np.complex128)
    ref = np.linalg.solve(A64, b64[..., None])[..., 0]
    err = np.linalg.norm(x - ref, axis=1) / np.linalg.norm(ref, axis=1)
    bound = 4 * N * 2.0 ** -23 * np.linalg.cond(A64)
    assert np.all(err <= bound), (err / bound).max()


def test_lu_nonfinite_stays_in_its_system():
    from cos_gb300 import capon
    rng = np.random.default_rng(5)
    for N in (8, 12, 32, 40):
        A = (rng.standard_normal((5, N, N)) + 1j * rng.standard_normal((5, N, N)) + 4 * np.eye(N)).astype(np.complex64)
        b = np.ones((5, N), np.complex64)
        clean = np.zeros((5, N), np.complex64)
        assert capon.Solver().solve(clean, A, b, N, 5) == 0
        A[2] = 0                     # singular: not finite
        A[3, 1, 2] = np.nan
        x = np.zeros((5, N), np.complex64)
        assert capon.Solver().solve(x, A, b, N, 5) == 0
        assert np.array_equal(x[[0, 1, 4]], clean[[0, 1, 4]])
        assert not np.isfinite(x[2]).all() and not np.isfinite(x[3]).all()
