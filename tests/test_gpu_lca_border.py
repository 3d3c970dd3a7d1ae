"""LCA selection where a filter's border covers whole tiles of the image, all of it or all but a few pixels, and where the
last chunk of windows is short: the border keeps zeros and window 0, the interior the oracle's choice."""
import numpy as np
import pytest

from test_gpu_lca_tiles import test_lca_tiles as check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Ny,Nx,Yf,Xf", [(16, 16, 255, 1), (100, 40, 101, 1), (101, 40, 101, 1), (40, 101, 1, 101),
                                         (130, 70, 101, 1), (50, 140, 1, 101), (33, 40, 15, 15), (3, 3, 5, 5)])
@pytest.mark.parametrize("Nw", [2, 4, 9, 12, 13])
def test_border(Ny, Nx, Nw, Yf, Xf):
    from cos_gb300 import lca
    if Ny >= Yf or Nx >= Xf:   # the oracle's slices need one of them
        check(Ny, Nx, Nw, Yf, Xf)
    Z = np.ones((Ny, Nx, Nw), np.complex64)
    img, win = lca.lca(Z, np.ones((Yf, Xf)))
    inner = np.zeros((Ny, Nx), bool)
    inner[Yf // 2:max(Ny - Yf // 2, 0), Xf // 2:max(Nx - Xf // 2, 0)] = True
    assert np.array_equal(img, np.where(inner, 1, 0)) and not win.any()
