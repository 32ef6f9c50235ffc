"""FLOP counters of the library against the products that it launches."""
import pytest

import ugacc_gb300 as U
from ugacc_gb300.generator import make_hamiltonian


@pytest.mark.gpu
@pytest.mark.parametrize("no,nv", [(2, 64), (4, 66)])
def test_products_of_the_mixed_triples(no, nv):
    """Three products for a tuple with two equal occupied indices, six for another, none for (i,i,i)."""
    h = make_hamiltonian(no, nv, seed=2)
    H = U.Hamiltonian(h.no, h.nv, h.fock, B=h.B)
    cc = U.CCWfn(H, {"R_CONVERGENCE": 1e-8, "PRECISION": "MIXED"})
    cc.compute_energy()
    H.ctx.reset_stats()
    cc.triples()
    tuples = [(i, j, k) for i in range(no) for j in range(i + 1) for k in range(j + 1) if k < i]
    products = sum(3 if i == j or j == k else 6 for i, j, k in tuples)
    assert H.ctx.stats()["tc_gemm_flops"] == 2.0 * products * nv ** 3 * (nv + no)


@pytest.mark.gpu
def test_ladder_counters():
    """One product per sweep, whatever the sweep that packs the integrals; ladder and Zmbij."""
    no, nv = 4, 40
    h = make_hamiltonian(no, nv, seed=3)
    H = U.Hamiltonian(h.no, h.nv, h.fock, B=h.B)
    cc = U.CCWfn(H, {"R_CONVERGENCE": 1e-8})
    for _ in range(2):
        H.ctx.reset_stats()
        cc.compute_energy()
        st = H.ctx.stats()
        assert st["ladder_launches"] == cc.iterations
        assert st["ladder_flops"] == cc.iterations * (2.0 * no ** 2 * nv ** 4 + 2.0 * no ** 3 * nv ** 3)
        assert st["ladder_bytes"] == cc.iterations * 8.0 * (nv ** 4 + 3 * no ** 2 * nv ** 2 + no * nv ** 3 + no ** 3 * nv)
        assert st["ladder_ms"] > 0
