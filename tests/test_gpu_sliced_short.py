"""Sliced FP64 GEMM with a short K (tc_gemm.cu, sliced_short_kernel) at the edges of its tiles,
K blocks and digit counts."""
import numpy as np
import pytest

import ugacc_gb300 as U

pytestmark = pytest.mark.gpu

# tiles of 128 x 32 and 128 x 64, K blocks of 64, the longest K (448) and the ring kernel after it
SHAPES = [(1, 1, 1), (127, 31, 63), (128, 32, 64), (129, 33, 65), (300, 64, 129), (257, 65, 256), (64, 97, 447),
          (200, 130, 448), (200, 130, 449), (20000, 16, 160), (1000, 1000, 16)]


@pytest.mark.parametrize("M,N,K", SHAPES)
@pytest.mark.parametrize("alpha,beta", [(1.0, 0.0), (-1.0, 1.0), (0.25, 1.0), (0.7, -0.3)])
def test_short_products(M, N, K, alpha, beta):
    rng = np.random.default_rng(M + 31 * N + K)
    A = rng.standard_normal((M, K)) * np.exp(2.0 * rng.standard_normal((M, 1)))
    B, C = rng.standard_normal((K, N)), rng.standard_normal((M, N))
    got = U.Context().gemm(A, B, C, alpha=alpha, beta=beta, precision=U.FP64_SLICED)
    ref = alpha * (A @ B) + beta * C
    # truncation at 9 x 6 bits, 14 2^(2-54) per term with the cross terms, over K terms at random signs
    scale = np.abs(A).max(axis=1)[:, None] * np.abs(B).max(axis=0)[None, :]
    assert np.all(np.abs(got - ref) <= 14 * 2.0 ** -52 * np.sqrt(K) * scale + 4 * 2.0 ** -53 * np.abs(ref)
                  + 2 * 2.0 ** -53 * np.abs(beta * C))


@pytest.mark.parametrize("digits", range(2, 10))
def test_short_products_by_digits(digits):
    """Whole numbers that the digits hold exactly (up to 2^(6d-2) per operand) multiply exactly."""
    rng = np.random.default_rng(digits)
    top = min(2 ** (6 * digits - 2), 2 ** 20)
    A, B = rng.integers(-top, top + 1, (150, 70)).astype(float), rng.integers(-top, top + 1, (70, 40)).astype(float)
    A[:, 0], B[0] = top, top  # every row's and column's scale
    got = U.Context().gemm(A, B, digits=digits)
    # products of digit order d and above are dropped: at most (d+1) 2^(-6(d+2)+10) of the scales' product, per term
    assert np.all(np.abs(got - A @ B) <= 70 * (digits + 1) * 2.0 ** (-6 * digits - 2) * (4.0 * top) ** 2)


def test_short_products_at_the_ends_of_the_range():
    rng = np.random.default_rng(8)
    A, B = rng.standard_normal((130, 50)), rng.standard_normal((50, 40))
    for sa, sb in ((2.0 ** 490, 2.0 ** 490), (2.0 ** -490, 2.0 ** -490), (2.0 ** -490, 2.0 ** -560), (0.0, 1.0)):
        got = U.Context().gemm(A * sa, B * sb, precision=U.FP64_SLICED)
        ref = (A * sa) @ (B * sb)
        scale = np.abs(A * sa).max(axis=1)[:, None] * np.abs(B * sb).max(axis=0)[None, :]
        # below 2^-500 a row's scale stays at 2^-500: its digits start lower
        floor = 2.0 ** -550 * np.abs(A * sa).max() * 50
        assert np.all(np.abs(got - ref) <= 1e-14 * np.sqrt(50) * scale + floor + 1e-320)
