"""The L = 16 candidates of four-warp CTAs (32-pixel tiles, three CTAs an SM) and the candidates with one row stride
for a range of channel counts: forced by name at the edges of their tiles and strides, with every output mode, equal to
the candidate they are chosen against (the same arithmetic per pixel, in another tile)."""
import pytest

pytestmark = pytest.mark.gpu


def outputs(x, L, K, rows, name, monkeypatch):
    import torch
    from cos_gb300 import capon
    monkeypatch.setenv("COS_CAPON_FUSED_CONFIG", name)
    Nx, out = x.shape[0], []
    for w, R in ((False, False), (True, False), (False, True)):
        f = capon.DeviceFrame(x=x, L=L, K=K, P=torch.empty((Nx, rows), device="cuda"))
        if w:
            f.w = torch.empty((Nx, rows, L), dtype=torch.complex64, device="cuda")
        if R:
            f.R = torch.empty((Nx, rows, L, L), dtype=torch.complex64, device="cuda")
        capon.capon_frames([f], capon.Context())
        out += [t for t in (f.z, f.P, f.w, f.R) if t is not None]
    torch.cuda.synchronize()
    return [torch.view_as_real(t) if t.is_complex() else t for t in out]


def check(L, K, M, rows, names, base, monkeypatch):
    import torch
    g = torch.Generator(device="cuda").manual_seed(M + rows)
    x = torch.randn((3, rows + 2 * K, M), dtype=torch.complex64, device="cuda", generator=g)
    want = outputs(x, L, K, rows, base, monkeypatch)
    for name in names:
        for a, b in zip(outputs(x, L, K, rows, name, monkeypatch), want):
            assert torch.equal(a, b), name


@pytest.mark.parametrize("M", [17, 32, 37, 40, 41, 48])
@pytest.mark.parametrize("K", [0, 1, 2])
@pytest.mark.parametrize("rows", [1, 31, 32, 33, 70])
def test_four_warp_candidates(rows, K, M, monkeypatch):
    T = 2 * K + 1
    names = [f"L16.G4.W4.N1.B3.T{T}"] + ([f"L16.G4.W4.N1.B3.M32.T{T}"] if M == 32 else [])
    names += [f"L16.G4.W4.N1.B3.X42.T{T}"] if M <= 40 else []
    check(16, K, M, rows, names, f"L16.G4.W8.N1.sync.T{T}", monkeypatch)


@pytest.mark.parametrize("M", [32, 33, 47, 63, 64])
@pytest.mark.parametrize("K", [0, 1, 2])
@pytest.mark.parametrize("rows", [1, 63, 65])
def test_stride_66_candidates(rows, K, M, monkeypatch):
    T = 2 * K + 1
    check(32, K, M, rows, [f"L32.G8.W8.N2.X66.T{T}"], f"L32.G8.W8.N2.sync.T{T}", monkeypatch)


@pytest.mark.parametrize("M", [48, 61, 97])
@pytest.mark.parametrize("K", [0, 1, 4])
@pytest.mark.parametrize("rows", [1, 23, 25])
def test_twelve_warp_l48(rows, K, M, monkeypatch):
    check(48, K, M, rows, ["L48.G16.W12.N1"], "L48.G16.W8.N1.sync", monkeypatch)
