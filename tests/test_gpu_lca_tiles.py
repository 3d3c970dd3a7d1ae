"""The one-pass LCA selection at the edges of its 32 x 16 pixel tiles: images smaller than a tile or one past it, long
filters either way, window counts that go in several chunks of shared memory.  The window must equal the FP64
oracle's except where its two best sums tie to the bound of the FP32 sums (n + 2 roundings each), the image exactly."""
import numpy as np
import pytest

import lca_oracle

pytestmark = pytest.mark.gpu

# Ny, Nx, Nw, Yf, Xf
CASES = [(1, 1, 1, 1, 1), (17, 33, 3, 1, 1), (16, 32, 8, 5, 1), (15, 31, 5, 3, 3), (33, 65, 2, 1, 5), (40, 70, 9, 7, 5),
         (48, 40, 33, 3, 3), (60, 35, 130, 5, 1), (300, 33, 3, 255, 1), (20, 300, 4, 1, 255), (34, 66, 40, 15, 15)]


@pytest.mark.parametrize("Ny,Nx,Nw,Yf,Xf", CASES)
def test_lca_tiles(Ny, Nx, Nw, Yf, Xf):
    from cos_gb300 import lca
    rng = np.random.default_rng(Ny * 7 + Nw)
    Z = (rng.standard_normal((Ny, Nx, Nw)) + 1j * rng.standard_normal((Ny, Nx, Nw))).astype(np.complex64)
    wrf = rng.uniform(0.5, 1.5, (Yf, Xf))
    img, win = lca.lca(Z, wrf)
    out = lca_oracle.lca(Z, wrf)
    same = win == out[1]
    if len(out) == 3:
        s = np.sort(out[2], axis=2)
        near = (s[..., 1] - s[..., 0] <= (Yf * Xf + 2) * 2.0 ** -23 * s[..., 0]) if Nw > 1 else np.zeros(win.shape, bool)
        assert not (~same & ~near).any()
    else:
        assert same.all()
    np.testing.assert_array_equal(img[same], out[0][same])
