"""Time-domain steering of few pixels (hydrophones shared by a CTA's warps) and of short beams (a warp's pixels on several
beams), cube and image, against the FP64 oracle with the bound of the tile tests."""
import numpy as np
import pytest

import tdib_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_h", [1, 3, 4, 5, 9, 17, 33, 64, 100, 256])
@pytest.mark.parametrize("n_x,n_y", [(1, 1), (33, 1), (7, 2), (2, 33), (400, 3)])
def test_few_pixels(n_h, n_x, n_y):
    from cos_gb300 import tdib
    s = tdib_oracle.scenario(seed=n_h + n_x, n_h=n_h, n_x=n_x, n_y=n_y)
    s["yarr"] = s["yarr"] + 0.01 * np.arange(n_x)[:, None]      # no two beams alike
    if n_x > 1:
        s["yarr"][-1] = 500.0                                   # past the time axis
    ref = tdib_oracle.steer(**s)
    Xd, img = tdib.steer(**s), tdib.tdib(**s)
    scale = np.nanmax(np.abs(ref))
    d = np.abs(s["x_r"]).max() + np.abs(s["x_r"]).mean() + np.abs(s["D"]).max()
    tol = 1e-5 + 4 * 2.0 ** -24 * d / s["c"] * (2 * np.pi * s["fc"] + 2 / (s["mtaxe"][1] - s["mtaxe"][0]))
    want = ref.sum(2).T / n_h
    for got, ex in ((Xd, ref), (img, want)):
        assert np.array_equal(np.isnan(got), np.isnan(ex))
        assert np.nanmax(np.abs(got - ex)) <= tol * scale
