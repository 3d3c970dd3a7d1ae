"""The general element-space path (subarray lengths without a fused kernel, long windows, forward-backward averaging;
exact products below 2.5 L snapshots): both sides of every padded length of its solve stage, windows with and without a compile-time row ring, odd channel
counts, partial tiles, L = M and one pixel, against the FP64 oracle at the fused bars (P 1e-4, z 1e-3 of sqrt(P),
w 2e-3; R to 1e-6 of its largest entry)."""
import numpy as np
import pytest

import oracle
from test_gpu_capon import assert_close

pytestmark = pytest.mark.gpu

# Nx, Ny, M, L, K, fb
CASES = [
    (3, 40, 5, 1, 1, 0), (2, 41, 7, 2, 0, 0), (3, 33, 16, 7, 2, 0), (2, 50, 17, 8, 1, 0), (2, 37, 18, 9, 1, 1),
    (2, 60, 31, 15, 3, 0), (2, 44, 37, 16, 3, 0), (2, 39, 33, 17, 1, 0), (2, 35, 46, 23, 2, 1), (2, 70, 48, 24, 2, 0),
    (2, 36, 52, 25, 4, 0), (2, 40, 62, 31, 1, 0), (3, 77, 64, 32, 2, 1), (2, 30, 72, 32, 2, 0), (2, 33, 67, 33, 0, 0),
    (2, 30, 81, 40, 1, 0), (1, 40, 95, 47, 2, 0), (1, 40, 96, 48, 1, 1), (1, 33, 99, 49, 1, 0), (1, 30, 126, 63, 3, 0),
    (1, 34, 128, 64, 4, 1), (2, 20, 24, 24, 1, 0), (1, 5, 40, 20, 2, 0), (1, 30, 21, 10, 12, 0),
    (2, 40, 31, 20, 1, 0), (2, 40, 30, 20, 1, 0), (1, 36, 200, 60, 1, 0), (40, 50, 60, 20, 1, 0),
]


def frame(Nx, Ny, M, seed):
    from cos_gb300 import synth
    if Ny > 30:
        return synth.cube(Ny, Nx, M, [10.0, 5.0], seed=seed)
    rng = np.random.default_rng(seed)
    return (rng.standard_normal((Nx, Ny, M)) + 1j * rng.standard_normal((Nx, Ny, M))).astype(np.complex64)


@pytest.mark.parametrize("want_w", [False, True])
@pytest.mark.parametrize("Nx,Ny,M,L,K,fb", CASES)
def test_general(Nx, Ny, M, L, K, fb, want_w):
    from cos_gb300 import capon
    x = frame(Nx, Ny, M, seed=M * 10 + K)
    z, P, w = capon.getCaponGPU(x, 0.01, L, K, None, bool(fb), want_w=want_w)
    ref = oracle.capon(x, 0.01, L, K, fb=bool(fb), nthreads=4)
    assert_close(z, P, w, ref, what=f"M{M} L{L} K{K} fb{fb}")


@pytest.mark.parametrize("layout", [0, 1])
@pytest.mark.parametrize("L,M,K", [(13, 27, 1), (24, 48, 2), (40, 77, 1)])
def test_general_R(L, M, K, layout):
    from cos_gb300 import capon
    Nx, Ny = 2, 34
    x = frame(Nx, Ny, M, seed=L)
    n = Ny - 2 * K
    z, P, R = np.zeros((Nx, n), np.complex64), np.zeros((Nx, n), np.float32), np.zeros((Nx, n, L, L), np.complex64)
    assert capon.Capon().getCaponEx(z, P, None, R, x, 0.01, L, K, M, Nx, Ny, 0, capon.opts(r_layout=layout)) == 0
    ref = oracle.capon(x, 0.01, L, K, want_R=True, nthreads=4)
    want = ref["R"] if layout else np.swapaxes(ref["R"], -1, -2) * ((M - L + 1) * (2 * K + 1))
    assert np.abs(R - want).max() <= 1e-6 * np.abs(want).max()
    assert_close(z, P, None, ref, what=f"R L{L}")


def test_beams_alone_and_absolute_loading():
    """A beam's outputs do not depend on the frame around it; absolute loading d on the normalised R."""
    from cos_gb300 import _lib, capon
    x = frame(5, 61, 41, seed=3)
    a = capon.getCaponGPU(x, 0.3, 20, 1, loading=_lib.LOAD_ABSOLUTE)
    ref = oracle.capon(x, 0.3, 20, 1, absolute=True, nthreads=4)
    assert_close(*a, ref, what="absolute")
    b = capon.getCaponGPU(x[2:3], 0.3, 20, 1, loading=_lib.LOAD_ABSOLUTE)
    assert np.abs(a[0][2:3] - b[0]).max() <= 1e-6 * np.abs(b[0]).max()
