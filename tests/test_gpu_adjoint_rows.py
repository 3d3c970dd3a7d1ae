"""The row-wise adjoint at the edges of its lane blocks: one subarray, blocks that do not divide the subarrays, more
items than lanes (several passes), long windows against few rows and in several launches, masked gradients, against FP64 torch.linalg autograd.
FP32 weights of a system of condition number up to about 1e3 carry about 1e-4; the bound is the adjoint's 1e-3."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# L, K, M, Ny, Nx
CASES = [(8, 0, 8, 5, 2), (8, 1, 21, 40, 3), (16, 3, 33, 20, 2), (16, 1, 32, 65, 2), (24, 2, 49, 33, 2), (24, 0, 71, 9, 1),
         (32, 2, 64, 40, 2), (32, 1, 67, 31, 2), (32, 4, 33, 10, 1), (32, 0, 32, 3, 1), (20, 1, 40, 40, 2),
         (32, 4, 128, 30, 2), (16, 17, 33, 60, 1), (32, 9, 64, 40, 1)]


@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("L,K,M,Ny,Nx", CASES)
def test_adjoint_rows(L, K, M, Ny, Nx, masked):
    import torch
    from cos_gb300 import autograd
    g = torch.Generator().manual_seed(L * 100 + M)
    x = torch.randn((Nx, Ny, M), dtype=torch.complex64, generator=g)
    tau = torch.rand(M, generator=g) * 0.1 - 0.05
    gP = torch.randn((Nx, Ny - 2 * K), generator=g)
    if masked:
        gP[:, ::3] = 0.0
        gP[0, : (Ny - 2 * K) // 2] = 0.0
    d = 0.2
    xs = x.cuda().requires_grad_(True)
    ts, ds = tau.cuda().requires_grad_(True), torch.tensor(d, device="cuda", requires_grad=True)
    P = autograd.capon_power(xs, ds, ts, L, K)
    gx, gt, gd = torch.autograd.grad(P, [xs, ts, ds], gP.cuda())
    x64 = x.to(torch.complex128).requires_grad_(True)
    t64, d64 = tau.double().requires_grad_(True), torch.tensor(float(np.float32(d)), dtype=torch.float64, requires_grad=True)
    P64 = autograd.capon_power_reference(x64, d64, t64, L, K).reshape(gP.shape)
    rx, rt, rd = torch.autograd.grad(P64, [x64, t64, d64], gP.double())
    for got, want in ((gx, rx), (gt, rt), (gd, rd)):
        err = (got.cpu().to(want.dtype) - want).abs().max() / want.abs().max().clamp(min=1e-30)
        assert float(err) <= 1e-3, float(err)
    # rows outside every window of a pixel with a gradient get exactly nothing
    hit = torch.zeros((Nx, Ny), dtype=torch.bool)
    for t in range(2 * K + 1):
        hit[:, t:t + gP.shape[1]] |= gP != 0
    assert float(gx.cpu()[~hit].abs().sum()) == 0.0
