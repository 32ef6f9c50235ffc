"""Operand passes of the tensor-core products (two bf16 parts, digit slices with their row maxima) at the edges
of their 32 x 64 tiles, both orders of the operands, and at the ends of the exponent range."""
import numpy as np
import pytest

import ugacc_gb300 as U

EPS2 = 2.0 ** -16  # two bf16 parts: the rest of an element is below 2^-17 of it, the product's below 2^-16


@pytest.fixture(scope="module")
def ctx():
    return U.Context()


def _operands(ctx_seed, M, N, K, ta, tb):
    r = np.random.default_rng(ctx_seed)
    A = r.standard_normal((M, K)) * np.exp2(r.integers(-9, 9, (M, 1)))
    B = r.standard_normal((K, N)) * np.exp2(r.integers(-9, 9, (1, N)))
    return A, B, np.ascontiguousarray(A.T) if ta else A, np.ascontiguousarray(B.T) if tb else B


@pytest.mark.gpu
@pytest.mark.parametrize("ta,tb", [(False, False), (True, True), (True, False)])
@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (31, 33, 63), (32, 32, 64), (33, 31, 65), (130, 70, 257), (65, 1, 1025)])
def test_products_at_tile_edges(ctx, M, N, K, ta, tb):
    A, B, a, b = _operands(M * 1000 + K, M, N, K, ta, tb)
    bound = np.abs(A) @ np.abs(B)
    split = ctx.gemm(a, b, transa=ta, transb=tb, precision=U.MIXED)
    # FP32 accumulation of K terms of three products beside the parts' rest
    assert np.all(np.abs(split - A @ B) <= (3 * EPS2 + 3 * K * 2.0 ** -24) * bound + 1e-300)
    sliced = ctx.gemm(a, b, transa=ta, transb=tb, digits=9)
    # nine digits of six bits against the row and column maxima, the dropped orders included
    scale = np.abs(A).max(1, keepdims=True) * np.abs(B).max(0, keepdims=True)
    assert np.all(np.abs(sliced - A @ B) <= 2.0 ** -40 * K * scale + 1e-15 * bound)


@pytest.mark.gpu
def test_split_at_the_ends_of_the_exponent_range(ctx):
    """One element per row against the identity: what an element becomes in two parts."""
    big = 3.0e38
    x = np.array([0.0, -0.0, 1.5, -2.0 ** -126, 2.0 ** -127, 1.75 * 2.0 ** -130, 2.0 ** -149, 2.0 ** -151, 5e-324, big,
                  -big])
    A = np.zeros((x.size, 16))
    A[:, 0] = x
    out = ctx.gemm(A, np.eye(16), precision=U.MIXED)
    assert np.all(np.abs(out[:, 0] - x) <= EPS2 * np.abs(x) + 2.0 ** -126)
    assert np.all(out[:, 1:] == 0.0)


@pytest.mark.gpu
def test_row_maxima_of_one_and_several_column_chunks(ctx):
    """A maximum in any chunk of columns: an integer row, exact in nine digits."""
    for K in (64, 511, 513, 5000):
        for pos in (0, K // 2, K - 1):
            A = np.ones((3, K))
            A[1, pos] = 2.0 ** 20
            out = ctx.gemm(A, np.ones((K, 2)), digits=9)
            np.testing.assert_array_equal(out, A @ np.ones((K, 2)))


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K", [(33, 32, 64), (130, 64, 40), (7, 66, 64), (129, 100, 128)])
def test_accumulating_product_by_sectors_and_by_elements(ctx, M, N, K):
    """C += A B: rows of C on 32-byte boundaries and not, whole and ragged blocks of 32 columns."""
    A, B, a, b = _operands(N, M, N, K, False, False)
    C = np.random.default_rng(N + 1).standard_normal((M, N))
    bound = np.abs(A) @ np.abs(B)
    out = ctx.gemm(a, b, C=C, beta=1.0, precision=U.MIXED)
    assert np.all(np.abs(out - (C + A @ B)) <= (3 * EPS2 + 3 * K * 2.0 ** -24) * bound + 1e-15 * np.abs(C))
