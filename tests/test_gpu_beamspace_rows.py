"""Beamspace with 5 < Nb <= 32 beams (the row-sharing kernel): the edges of its lane groups (8, 16, 32 lanes per
pixel), odd beam counts, partial tiles, windows longer than a tile's halo, and the first sizes it leaves to the
warp kernel, against the FP64 oracle at the fused bar (P 1e-4, z 1e-3 of sqrt(P), w 2e-3)."""
import numpy as np
import pytest

import oracle
from test_gpu_capon import assert_close

pytestmark = pytest.mark.gpu

# Nx, Ny, M, L, K, Nb
CASES = [
    (2, 40, 24, 12, 1, 6),     # narrowest beam count
    (3, 70, 64, 32, 1, 8),     # a full group of 8 lanes, a partial last tile
    (2, 33, 33, 17, 0, 9),     # odd everything, one window row
    (2, 41, 48, 24, 2, 16),    # a full group of 16 lanes
    (2, 35, 51, 29, 1, 17),    # group of 32, one past 16
    (1, 30, 64, 33, 1, 32),    # a full group of 32 lanes (an even Nb = L repeats a DFT bin: no solution)
    (2, 60, 20, 10, 12, 7),    # a window longer than the tile
    (1, 5, 40, 20, 2, 11),     # one pixel
    (1, 12, 40, 36, 0, 33),    # past the kernel: one warp per pixel
]


@pytest.mark.parametrize("loading", [0, 1, 2])
@pytest.mark.parametrize("Nx,Ny,M,L,K,Nb", CASES)
def test_beamspace_rows(Nx, Ny, M, L, K, Nb, loading):
    from cos_gb300 import capon, synth
    rng = np.random.default_rng(M * 100 + Nb)
    if Ny > 30:
        x = synth.cube(Ny, Nx, M, [10.0, 5.0], seed=M + Nb)
    else:
        x = (rng.standard_normal((Nx, Ny, M)) + 1j * rng.standard_normal((Nx, Ny, M))).astype(np.complex64)
    d = 0.5 if loading == 2 else 0.01
    z, P, w = capon.getCaponGPU(x, d, L, K, np.zeros((Nb, L)), loading=loading)
    if loading == 2:
        # B (R + d I) B^H = B R B^H + d I: relative loading restated per pixel
        ref = absolute(x, d, L, K, Nb)
    else:
        ref = oracle.capon(x, d, L, K, Nb=Nb, bs_loading=bool(loading), nthreads=4)
    assert_close(z, P, w, ref, what=f"M{M} L{L} K{K} Nb{Nb} load{loading}")


def absolute(x, d, L, K, Nb):
    Nx, Ny, M = x.shape
    Ns, T, n = M - L + 1, 2 * K + 1, Ny - 2 * K
    b = np.arange(Nb)
    bins = np.where(b > Nb // 2, b + (L - 2 * (Nb // 2) - 1), b)
    B = np.exp(-2j * np.pi * np.outer(bins, np.arange(L)) / L) / np.sqrt(L)
    xd = x.astype(np.complex128)
    z, P, w = np.zeros((Nx, n), complex), np.zeros((Nx, n)), np.zeros((Nx, n, L), complex)
    for i in range(Nx):
        for p in range(n):
            sub = np.lib.stride_tricks.sliding_window_view(xd[i, p:p + T], L, axis=1)   # T, Ns, L
            y = (sub.reshape(-1, L) @ B.T)
            R = y.T @ y.conj() / (Ns * T) + d * np.eye(Nb)
            a = B.sum(1)
            v = np.linalg.solve(R, a)
            den = (a.conj() @ v).real
            w[i, p] = B.conj().T @ v / den
            P[i, p] = 1.0 / den
            z[i, p] = w[i, p].conj() @ sub[K].mean(0)
    return dict(z=z, P=P, w=w)
