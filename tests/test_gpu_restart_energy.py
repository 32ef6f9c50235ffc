"""A CCSD solve that its starting amplitudes already satisfy: one sweep, and their energy."""
import numpy as np
import pytest

import ugacc_gb300 as U
from ugacc_gb300.generator import make_hamiltonian


@pytest.mark.gpu
@pytest.mark.parametrize("diis", [True, False])
def test_energy_of_a_solve_that_starts_converged(diis):
    h = make_hamiltonian(3, 9, seed=4)
    ints = h.ints_physicist()
    H = U.Hamiltonian(h.no, h.nv, h.fock, ints=ints)
    cc = U.CCWfn(H, {"R_CONVERGENCE": 1e-11, "MAXITER": 100, "DIIS": diis})
    cc.compute_energy()
    t1, t2 = cc.t1, cc.t2
    H.ctx.set("t1", t1)
    H.ctx.set("t2", t2)
    again = U.CCWfn(H, {"R_CONVERGENCE": 1e-8, "DIIS": diis})
    e = again.compute_energy()
    assert again.iterations == 1
    V = ints[:3, :3, 3:, 3:]  # the Fock matrix is diagonal: no one-electron term
    tau, L = t2 + np.einsum("ia,jb->ijab", t1, t1), 2.0 * V - V.swapaxes(2, 3)
    # one sum of the same terms in two orders, each a few roundings away
    assert abs(e - (tau * L).sum()) <= 2.0 ** -52 * (4 + tau.size ** 0.5) * (np.abs(tau) * np.abs(L)).sum()
