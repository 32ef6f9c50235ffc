"""Length of the FP32 accumulations of the split product (tc_gemm.cu, accumulation_blocks): operands of one sign,
whose sums the tensor core truncates at every step."""
import numpy as np
import pytest

import ugacc_gb300 as U

# (M, N, K, elements that one accumulation may cover): K in parts behind each other in C or through partial
# products, whole and ragged rows of C, one part only
CASES = [(2560, 2560, 2560, 896), (15440, 136, 12880, 2624), (7020, 91, 6903, 896), (160, 160, 40960, 576),
         (1521, 1521, 1521, 768), (4864, 512, 2048, 1024), (300, 200, 512, 256), (4000, 3000, 700, 700)]


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K,length", CASES)
@pytest.mark.parametrize("alpha,beta", [(1.0, 0.0), (-0.5, 1.0)])
def test_truncation_of_one_accumulation(M, N, K, length, alpha, beta):
    rng = np.random.default_rng(M + K)
    A, B = rng.random((M, K)), rng.random((K, N))
    C = alpha * K * rng.random((M, N)) if beta else None
    out = U.Context().gemm(A, B, C, alpha=alpha, beta=beta, precision=U.MIXED)
    got = (out - beta * C if beta else out) / alpha
    # the sum of all elements of A B.  3 length / 16 products are added to a sum that grows to its end, half of it on
    # average, each add truncated: half of the last place is lost on average, at most 2^-24 of the sum.  2^-21 for
    # the parts' rest, whose signs are mixed.
    exact = A.sum(0) @ B.sum(1)
    assert abs(got.sum() - exact) <= (3 * length / 16 * 2.0 ** -25 + 2.0 ** -21) * exact
