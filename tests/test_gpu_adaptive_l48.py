"""Adaptive refinement at L = 48, whose kernel keeps its warps in step with CTA barriers: tiles in which some warps'
pixels take the refinement pass and others' do not.  Every pixel must equal the plain or the refined result, the
ill-conditioned ones among them refined."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("want_w", [False, True])
@pytest.mark.parametrize("K,M,Ny", [(1, 96, 120), (1, 102, 61), (2, 96, 75)])
def test_some_warps_refine(K, M, Ny, want_w):
    from cos_gb300 import _lib, capon
    L, Nx, d = 48, 3, 1e-3
    rng = np.random.default_rng(M + Ny)
    x = (rng.standard_normal((Nx, Ny, M)) + 1j * rng.standard_normal((Nx, Ny, M))).astype(np.complex64)
    # a strong echo in single range rows, a window (2K+1 pixels) apart from the next
    ramp = np.exp(2j * np.pi * np.arange(M) / M).astype(np.complex64)
    for y in range(4, Ny, 11):
        x[:, y] += np.float32(300.0) * ramp

    def run(refine):
        o = capon.opts(refine=refine)
        n = Ny - 2 * K
        z, P = np.zeros((Nx, n), np.complex64), np.zeros((Nx, n), np.float32)
        w = np.zeros((Nx, n, L), np.complex64) if want_w else None
        assert capon.Capon().getCaponEx(z, P, w, None, x, d, L, K, M, Nx, Ny, 0, o) == 0
        return z, P, w

    plain, full, adapt = run(0), run(_lib.REFINE_ALL), run(_lib.REFINE_ADAPTIVE)
    ref = oracle.capon(x, d, L, K, nthreads=4)
    err = np.abs(adapt[1] - ref["P"]) / ref["P"]
    assert err.max() <= 1e-4, err.max()
    near = np.zeros(adapt[1].shape, bool)
    for y in range(4, Ny, 11):
        near[:, max(0, y - 2 * K):y + 1] = True
    # the two pixels of a warp take the pass together; a last one without a partner has a stale one
    n = near.shape[1]
    for p in range(0, n, 2):
        near[:, p:p + 2] = near[:, p:p + 2].any() or p + 1 == n
    # away from the echoes the plain result, bit for bit; beside them as near as the refined one
    assert np.array_equal(adapt[1][~near], plain[1][~near]) and np.array_equal(adapt[0][~near], plain[0][~near])
    e_full = np.abs(full[1] - ref["P"]) / ref["P"]
    assert err[near].max() <= max(2e-6, 4 * e_full[near].max())
    if want_w:
        ew = np.linalg.norm(adapt[2] - ref["w"], axis=-1) / np.linalg.norm(ref["w"], axis=-1)
        assert ew.max() <= 2e-3
