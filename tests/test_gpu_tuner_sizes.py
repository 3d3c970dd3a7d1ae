"""The autotuner's choice and the size of the launch that it was made on: a choice made on a short line is made again for
a full frame, whose times tell the candidates apart, and kept from there for frames of any size."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_choice_of_a_line_is_not_kept_for_a_frame(capfd, monkeypatch):
    import torch
    from cos_gb300 import capon
    monkeypatch.setenv("COS_CAPON_TUNE_VERBOSE", "1")
    monkeypatch.delenv("COS_CAPON_FUSED_CONFIG", raising=False)
    ctx = capon.Context()
    M, L, K = 32, 16, 1

    def run(Nx, Ny):
        x = torch.randn((Nx, Ny, M), dtype=torch.complex64, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
        f = capon.DeviceFrame(x=x, L=L, K=K, d=0.01, Nb=0, z=torch.empty((Nx, Ny - 2 * K), dtype=torch.complex64, device="cuda"),
                              P=torch.empty((Nx, Ny - 2 * K), dtype=torch.float32, device="cuda"))
        capfd.readouterr()
        capon.capon_frames([f], ctx=ctx)
        torch.cuda.synchronize()
        return capfd.readouterr().err.count("] tune "), f.P.cpu().numpy()

    first, line = run(1, 64)
    assert first >= 2
    assert run(1, 64)[0] == 0
    assert run(3, 64)[0] == 0                # up to four times as many pixels
    assert run(128, 1024)[0] == first        # a full frame
    assert run(200, 2048)[0] == 0
    again, after = run(1, 64)
    assert again == 0
    np.testing.assert_allclose(after, line, rtol=1e-5)
