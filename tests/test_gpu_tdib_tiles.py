"""Time-domain steering at the edges of its tiles (32 range pixels a warp, 16 hydrophones a transposed tile), cube and
image together and alone, with delays before and past the time axis, against the FP64 oracle.  The bound follows from
the FP32 corrections: the carrier phase fc d / c of a receiver at distance d from the origin carries a few roundings of
its own size, and the interpolation weight those of d / (c dt)."""
import numpy as np
import pytest

import tdib_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_h,n_x,n_y", [(1, 3, 1), (3, 2, 31), (15, 2, 32), (16, 1, 33), (17, 9, 65), (64, 5, 100),
                                         (255, 2, 40), (256, 3, 7)])
def test_tdib_tiles(n_h, n_x, n_y):
    from cos_gb300 import tdib
    s = tdib_oracle.scenario(seed=n_h, n_h=n_h, n_x=n_x, n_y=n_y)
    if n_y > 2:   # the first pixel far before the time axis, the last far past it
        s["yarr"][:, 0] = 0.5
        s["yarr"][:, -1] = 500.0
    ref = tdib_oracle.steer(**s)
    Xd = tdib.steer(**s)
    img = tdib.tdib(**s)
    scale = np.nanmax(np.abs(ref))
    d = np.abs(s["x_r"]).max() + np.abs(s["x_r"]).mean() + np.abs(s["D"]).max()
    tol = 1e-5 + 4 * 2.0 ** -24 * d / s["c"] * (2 * np.pi * s["fc"] + 2 / (s["mtaxe"][1] - s["mtaxe"][0]))
    assert np.array_equal(np.isnan(Xd), np.isnan(ref.astype(np.complex64)))
    assert np.nanmax(np.abs(Xd - ref)) <= tol * scale
    want = ref.sum(2).T / n_h
    assert np.array_equal(np.isnan(img), np.isnan(want))
    assert np.nanmax(np.abs(img - want)) <= tol * scale
