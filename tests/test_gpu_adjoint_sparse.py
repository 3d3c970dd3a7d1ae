"""The adjoint with gradients at few pixels: rows without any are left out, windows in one and in several passes (a last
one shorter than the others among them), weights that are not finite where the gradient is zero, against the adjoint's
formula in FP64.  Bound: each entry is a sum of at most L T products of a sum of L products, in FP32."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def adjoint64(x, w, gP, L, K):
    Nx, Ny, M = x.shape
    T, Ns = 2 * K + 1, M - L + 1
    x, w = x.astype(np.complex128), np.where(gP[..., None] != 0, w, 0).astype(np.complex128)
    gx, gd = np.zeros(x.shape, complex), 0.0
    for b, p in zip(*np.nonzero(gP)):
        gd += gP[b, p] * np.sum(np.abs(w[b, p]) ** 2)
        for t in range(T):
            e = np.lib.stride_tricks.sliding_window_view(x[b, p + t], L) @ w[b, p].conj() * gP[b, p] / (Ns * T)
            gx[b, p + t] += np.convolve(e, w[b, p])
    return gx, gd, 2 * (gx.real * x.imag - gx.imag * x.real).sum((0, 1))


@pytest.mark.parametrize("density", [0.0, 0.01, 0.2, 1.0])
@pytest.mark.parametrize("Nx,n,M,L,K", [(3, 70, 33, 16, 1), (2, 40, 128, 32, 9), (1, 9, 50, 32, 17), (5, 300, 17, 8, 2),
                                        (2, 50, 64, 24, 20), (2, 33, 40, 20, 1)])
def test_sparse(Nx, n, M, L, K, density):
    import torch
    from cos_gb300 import _lib, capon
    rng = np.random.default_rng(M + K)
    noise = lambda *s: (rng.standard_normal(s) + 1j * rng.standard_normal(s)).astype(np.complex64)
    x, w = noise(Nx, n + 2 * K, M), noise(Nx, n, L)
    gP = (rng.standard_normal((Nx, n)) * (rng.random((Nx, n)) < density)).astype(np.float32)
    w[gP == 0] = np.nan
    dev = lambda v: torch.from_numpy(v).cuda()
    xd, wd, gd_ = dev(x), dev(w), dev(gP)
    gx, gd, gt = torch.zeros_like(xd), torch.zeros(1, device="cuda"), torch.zeros(M, device="cuda")
    ctx = capon.Context()
    a = _lib.Adjoint(xd.data_ptr(), wd.data_ptr(), gd_.data_ptr(), gx.data_ptr(), gd.data_ptr(), gt.data_ptr(), L, K, M,
                     Nx, n + 2 * K)
    assert _lib.lib.cos_capon_backward(ctx.handle, ctypes.byref(a), torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    rx, rd, rt = adjoint64(x, w, gP, L, K)
    eps = 2.0 ** -23
    size = np.abs(rx).max() + 1e-30
    assert np.abs(gx.cpu().numpy() - rx).max() <= 8 * np.sqrt(2 * L) * eps * np.sqrt(2 * K + 1) * size
    assert np.all(gx.cpu().numpy()[rx == 0] == 0)
    many = 1 + np.count_nonzero(gP)
    assert abs(float(gd) - rd) <= 4 * eps * np.sqrt(many * L) * np.sum(np.abs(gP)) * L * 2 + 1e-30
    assert np.abs(gt.cpu().numpy() - rt).max() <= 16 * eps * np.sqrt(2 * L * many) * size * np.abs(x).max() * np.sqrt(x.size / M) + 1e-30
