"""Element-space frames without a fused instantiation: windows whose samples, four pixels of them, exceed a CTA's shared
memory are refused, with and without refinement, and the longest ones within it are served."""
import numpy as np
import pytest

import oracle
from test_gpu_capon import assert_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fb", [False, True])
@pytest.mark.parametrize("refine", [0, 1])
@pytest.mark.parametrize("M,L,K", [(300, 32, 16), (240, 60, 16), (48, 24, 76)])
def test_refused(M, L, K, fb, refine):
    from cos_gb300 import capon
    assert 32 * (2 * K + 1) * M > 227 * 1024
    x = np.ones((1, 2 * K + 3, M), np.complex64)
    with pytest.raises(capon.CaponError) as e:
        capon.getCaponGPU(x, 0.01, L, K, None, fb, refine=refine)
    assert e.value.status == 801


@pytest.mark.parametrize("refine", [0, 1])
@pytest.mark.parametrize("M,L,K", [(300, 32, 11), (48, 24, 75), (20, 10, 181)])
def test_longest_served(M, L, K, refine):
    from cos_gb300 import capon
    assert 32 * (2 * K + 1) * M <= 227 * 1024 < 32 * (2 * K + 3) * M
    rng = np.random.default_rng(M)
    x = (rng.standard_normal((2, 2 * K + 5, M)) + 1j * rng.standard_normal((2, 2 * K + 5, M))).astype(np.complex64)
    ref = oracle.capon(x, 0.01, L, K, nthreads=4)
    assert_close(*capon.getCaponGPU(x, 0.01, L, K, refine=refine), ref, what=f"M{M} L{L} K{K}")
