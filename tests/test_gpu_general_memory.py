"""The host-pointer call counts what a general frame needs: its records, about half of R, and not the buffers of the
pipeline that holds R twice.  The device's memory is taken up to a rest that lies between the two."""
import numpy as np
import pytest

import oracle
from test_gpu_capon import assert_close

pytestmark = pytest.mark.gpu


def test_host_call_in_little_memory():
    import torch
    from cos_gb300 import capon
    Nx, Ny, M, L = 32, 400, 80, 40
    n = Nx * Ny
    rng = np.random.default_rng(3)
    x = (rng.standard_normal((Nx, Ny, M)) + 1j * rng.standard_normal((Nx, Ny, M))).astype(np.complex64)
    z, P = np.zeros((Nx, Ny), np.complex64), np.zeros((Nx, Ny), np.float32)
    records, pipeline = n * 8 * (L * (L + 2) // 2 + L + 2), n * 8 * (2 * L * L + L)
    frame = n * (8 * M + 12)
    assert records + frame + (64 << 20) < pipeline
    warm = capon.Capon()                # module and local memory are there before the rest is measured
    args = (0.01, L, 0, M, 1, Ny, 0)
    assert warm.getCaponEx(z[:1], P[:1], None, None, x[:1], *args) == 0
    warm.close()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    rest = records + frame + (48 << 20)
    ballast = torch.empty(torch.cuda.mem_get_info()[0] - rest, dtype=torch.uint8, device="cuda")
    try:
        ctx = capon.Capon()
        status = ctx.getCaponEx(z, P, None, None, x, 0.01, L, 0, M, Nx, Ny, 0)
        ctx.close()
    finally:
        del ballast
        torch.cuda.empty_cache()
    assert status == 0
    ref = oracle.capon(x[:2], 0.01, L, 0, nthreads=4)
    assert_close(z[:2], P[:2], None, ref, what="little memory")
