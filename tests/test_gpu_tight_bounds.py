"""Products of the mixed form against bounds close to what their digits and parts give: lengths and widths at the
edges of the short-K kernel's tiles (16, 32 and 48 columns, K blocks of 64, K up to 448), the operand passes' tiles, a
single column in several passes over K, and (T) energies where every tuple takes half its products."""
import numpy as np
import pytest

import ugacc_gb300 as U
from ugacc_gb300.generator import make_hamiltonian

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    return U.Context()


def _check_nine_digits(ctx, M, N, K, seed, **kw):
    rng = np.random.default_rng(seed)
    A = rng.standard_normal((M, K)) * np.exp2(rng.integers(-9, 9, (M, 1)))
    B = rng.standard_normal((K, N)) * np.exp2(rng.integers(-9, 9, (1, N)))
    got = ctx.gemm(A.T if kw.get("transa") else A, B.T if kw.get("transb") else B, digits=9, **kw)
    ref = A @ B
    # 9 x 6 bits of the row and column maxima, 14 2^(2-54) per term with the cross terms, K terms at random signs,
    # and the roundings of result and reference
    scale = np.abs(A).max(1)[:, None] * np.abs(B).max(0)[None, :]
    assert np.all(np.abs(got - ref) <= 14 * 2.0 ** -52 * np.sqrt(K) * scale + 4 * 2.0 ** -53 * np.abs(ref))


@pytest.mark.parametrize("N", [15, 16, 17, 47, 48, 49, 95, 96, 97])
@pytest.mark.parametrize("K", [1, 64, 65, 448])
def test_short_products_at_column_tiles(ctx, N, K):
    _check_nine_digits(ctx, 130, N, K, 100 * N + K)


@pytest.mark.parametrize("ta,tb", [(False, False), (True, True), (True, False)])
@pytest.mark.parametrize("M,N,K", [(31, 33, 63), (33, 31, 65), (130, 70, 257), (65, 1, 1025), (129, 257, 700)])
def test_sliced_products_at_operand_tiles(ctx, M, N, K, ta, tb):
    _check_nine_digits(ctx, M, N, K, M + K, transa=ta, transb=tb)


@pytest.mark.parametrize("M,N,K,length", [(5000, 1, 20000, 1344), (129, 1, 70000, 960)])
def test_one_column_in_parts_of_k(ctx, M, N, K, length):
    rng = np.random.default_rng(K)
    A, B = rng.random((M, K)), rng.random((K, N))
    out, exact = ctx.gemm(A, B, precision=U.MIXED), A.sum(0) @ B.sum(1)
    # truncated accumulations over `length` elements (accumulation_blocks: 15 and 73 parts): at most 2^-25 of the sum
    # for each of 3 length / 16 products on average; the parts' rest has mixed signs
    assert abs(out.sum() - exact) <= (3 * length / 16 * 2.0 ** -25 + 2.0 ** -21) * exact


@pytest.mark.parametrize("no,nv", [(2, 64), (2, 65), (2, 66), (2, 71), (2, 96), (3, 68)])
def test_mixed_triples_from_half_their_products(no, nv):
    """no = 2: (1,0,0) and (1,1,0) only.  Errors of 2^-17 in the elements of W3, independent over the nv^3 / 6 terms,
    in a sum that cancels to a tenth of its terms: 2 2^-17 10 sqrt(6 / nv^3) = 7e-7 of the energy at nv = 64.  1e-5 is
    ten of those; one 8 x 8 x 8 tile without its exchange is 1/500 of the terms."""
    h = make_hamiltonian(no, nv, seed=7 * no + nv)
    H = U.Hamiltonian(h.no, h.nv, h.fock, B=h.B)
    cc = U.CCWfn(H, {"R_CONVERGENCE": 1e-11, "MAXITER": 100})
    cc.compute_energy()
    e64 = cc.triples()
    mixed = U.CCWfn(H, {"R_CONVERGENCE": 1e-11, "MAXITER": 100, "PRECISION": "MIXED"}).triples()
    assert abs(mixed - e64) < 1e-5 * abs(e64)
