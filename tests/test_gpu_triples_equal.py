"""(T) with few occupied orbitals, where most tuples have two equal indices and so half the products, against
the oracle, at the edges of the 32 x 32 tiles of the exchange pass."""
import pytest

import ugacc_gb300 as U
from oracle import cc as O
from ugacc_gb300.generator import make_hamiltonian


@pytest.mark.gpu
@pytest.mark.parametrize("no,nv", [(1, 6), (2, 2), (2, 31), (2, 33), (3, 32), (3, 65), (4, 20)])
def test_triples_of_few_occupied(no, nv):
    h = make_hamiltonian(no, nv, seed=100 * no + nv)
    H = U.Hamiltonian(h.no, h.nv, h.fock, B=h.B)
    cc = U.CCWfn(H, {"R_CONVERGENCE": 1e-11, "MAXITER": 100})
    cc.compute_energy()
    ref = O.CCWfn(O.Hamiltonian(h), maxiter=100, r_convergence=1e-11)
    ref.compute_energy()
    # both sides' amplitudes are within some 1e-11 of the solution, and (T) is quadratic in
    # them: 2 |E(T)| 1e-11 / |t|, below 1e-10 for these energies
    assert abs(cc.triples() - ref.tcorr_tjl()) < 1e-10


@pytest.mark.gpu
@pytest.mark.parametrize("no,nv", [(2, 64), (2, 66), (3, 68), (3, 71)])
def test_mixed_triples_of_few_occupied(no, nv):
    """The mixed form's half sets of products and the exchange in both energy kernels (nv % 4 == 0 or not)."""
    h = make_hamiltonian(no, nv, seed=100 * no + nv)
    H = U.Hamiltonian(h.no, h.nv, h.fock, B=h.B)
    cc = U.CCWfn(H, {"R_CONVERGENCE": 1e-11, "MAXITER": 100})
    cc.compute_energy()
    e64 = cc.triples()
    mixed = U.CCWfn(H, {"R_CONVERGENCE": 1e-11, "MAXITER": 100, "PRECISION": "MIXED"}).triples()
    # two bf16 parts leave 2^-16 of a product; the energy's sums of W V cancel to a tenth or so
    assert abs(mixed - e64) < 1e-3 * abs(e64)
