"""FP64 GEMM (dgemm.cu) at the edges of its patches, tiles, stages and K splits."""
import numpy as np
import pytest

import ugacc_gb300 as U

pytestmark = pytest.mark.gpu

# 8 x 4 patches, 16 x 16 and 32 x 32 tiles, K stages of 16 and 32, K over the CTAs of a cluster
# (ranges that leave the last ones empty or ragged) and over partial products in memory
SHAPES = [(1, 2, 1), (8, 4, 3), (9, 5, 33), (7, 3, 31), (16, 16, 8), (17, 15, 64), (25, 25, 361), (31, 33, 65),
          (33, 31, 129), (95, 19, 95), (2, 300, 17), (300, 2, 18), (16, 16, 8200), (3, 5, 70001), (65, 63, 4099),
          (1000, 37, 16), (2048, 160, 5), (513, 257, 100)]


@pytest.mark.parametrize("M,N,K", SHAPES)
@pytest.mark.parametrize("ta,tb", [(False, False), (True, False), (False, True), (True, True)])
def test_fp64_gemm_edges(M, N, K, ta, tb):
    rng = np.random.default_rng(M * 7919 + N * 31 + K)
    A, B, C = rng.standard_normal((M, K)), rng.standard_normal((K, N)), rng.standard_normal((M, N))
    ctx = U.Context()
    out = ctx.gemm(A.T if ta else A, B.T if tb else B, C=C, alpha=-0.5, beta=2.0, transa=ta, transb=tb)
    ref = -0.5 * (A @ B) + 2.0 * C
    # any order of summation: gamma_(K+2) (|A||B| + 2|C|) on either side
    bound = 2 * (K + 2) * 2.0 ** -53 * (0.5 * np.abs(A) @ np.abs(B) + 2.0 * np.abs(C))
    assert np.all(np.abs(out - ref) <= bound)


def test_fp64_gemm_nonfinite_stay_in_their_rows():
    rng = np.random.default_rng(3)
    A, B = rng.standard_normal((37, 50)), rng.standard_normal((50, 21))
    A[5, 7], B[3, 20] = np.nan, np.inf
    out = U.Context().gemm(A, B)
    ref = A @ B
    assert np.array_equal(np.isnan(out), np.isnan(ref)) and np.array_equal(np.isinf(out), np.isinf(ref))
    fine = np.isfinite(ref)
    assert np.allclose(out[fine], ref[fine], rtol=0, atol=1e-13)


@pytest.mark.parametrize("M,N,K", [(16, 16, 40000), (40, 9, 30000), (95, 95, 95)])
def test_split_products_repeat_and_are_timed(M, N, K):
    """The split's tickets come back to zero: a second product is the first one bit for bit; short
    products are timed by their own CTAs."""
    rng = np.random.default_rng(K)
    A, B = rng.standard_normal((M, K)), rng.standard_normal((K, N))
    ctx = U.Context()
    first = ctx.gemm(A, B)
    ctx.reset_stats()
    assert np.array_equal(ctx.gemm(A, B), first)
    st = ctx.stats()
    assert st["fp64_gemm_launches"] == 1 and st["fp64_gemm_flops"] == 2.0 * M * N * K
    assert 1e-4 < st["fp64_gemm_ms"] < 50.0
