"""Time-domain steering: delays that fall on the last sample of the time axis, which lies inside it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_last_sample():
    """One hydrophone at the origin and c = 1: a pixel at range t/2 has the delay t exactly."""
    from cos_gb300 import tdib
    fs, checked = 5e4, 0
    for n in range(600, 1000):
        t = np.arange(n) / fs
        dt = (t[-1] - t[0]) / (n - 1)
        if t[-1] / dt != n - 1 or not t[-1] * (1.0 / dt) > n - 1:
            continue
        mf = (np.arange(n) + 1.0 + 0.5j)[None].astype(np.complex64)
        Xd = tdib.steer(mf, t, np.zeros(1), np.zeros(1), 1.0, 0.0, np.zeros((1, 1)), np.full((1, 1), t[-1] / 2))
        assert Xd[0, 0, 0] == mf[0, -1]
        checked += 1
    assert checked >= 5
