"""The L = 16 candidates of four-warp CTAs (32-pixel tiles, three CTAs an SM): forced by name at the edges of their
tiles, with odd and even channel counts and every output mode, bit-equal to the eight-warp candidate they are chosen
against (the same arithmetic per pixel, in another tile)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [17, 32, 37, 48])
@pytest.mark.parametrize("K", [0, 1, 2])
@pytest.mark.parametrize("rows", [1, 31, 32, 33, 70])
def test_four_warp_candidates(rows, K, M, monkeypatch):
    import torch
    from cos_gb300 import capon
    T, Nx = 2 * K + 1, 3
    g = torch.Generator(device="cuda").manual_seed(M + rows)
    x = torch.randn((Nx, rows + 2 * K, M), dtype=torch.complex64, device="cuda", generator=g)

    def run(name):
        monkeypatch.setenv("COS_CAPON_FUSED_CONFIG", name)
        out = []
        for w, R in ((False, False), (True, False), (False, True)):
            f = capon.DeviceFrame(x=x, L=16, K=K, P=torch.empty((Nx, rows), device="cuda"))
            if w:
                f.w = torch.empty((Nx, rows, 16), dtype=torch.complex64, device="cuda")
            if R:
                f.R = torch.empty((Nx, rows, 16, 16), dtype=torch.complex64, device="cuda")
            capon.capon_frames([f], capon.Context())
            out += [t for t in (f.z, f.P, f.w, f.R) if t is not None]
        torch.cuda.synchronize()
        return out

    want = run(f"L16.G4.W8.N1.sync.T{T}")
    names = [f"L16.G4.W4.N1.B3.T{T}"] + ([f"L16.G4.W4.N1.B3.M32.T{T}"] if M == 32 else [])
    for name in names:
        for a, b in zip(run(name), want):
            assert torch.equal(torch.view_as_real(a) if a.is_complex() else a,
                               torch.view_as_real(b) if b.is_complex() else b), name
