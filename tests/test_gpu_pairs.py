"""The tile passes of pairs.cu at the edges of their 32 x 32 tiles and pair ranges: CCSD energies
and amplitudes, HBAR ladders (Lambda) and batches against the oracle."""
import numpy as np
import pytest

import ugacc_gb300 as U
from oracle import cc as O
from ugacc_gb300.generator import make_hamiltonian

pytestmark = pytest.mark.gpu

# no = 1 (no strict occupied pairs), nv = 1 (no strict virtual pairs), below, at and above a tile
SIZES = [(1, 1), (1, 5), (2, 1), (1, 33), (2, 31), (2, 32), (3, 33), (2, 65)]


def _oracle(h):
    cc = O.CCWfn(O.Hamiltonian(h), r_convergence=1e-10)
    cc.compute_energy()
    return cc


@pytest.mark.parametrize("no,nv", SIZES)
def test_ccsd_and_lambda_at_tile_edges(no, nv):
    h = make_hamiltonian(no, nv, 40 + no + nv)
    ref = _oracle(h)
    H = U.Hamiltonian.from_synthetic(h)
    cc = U.CCWfn(H, {"R_CONVERGENCE": 1e-10})
    cc.compute_energy()
    # both converged to |R| < 1e-10: amplitudes within |R| / |D| <= 1e-10 (|D| >= 1 here) of the solution
    assert abs(cc.eccsd - ref.eccsd) < 1e-10 and np.abs(cc.t2 - ref.t2).max() < 2e-10
    lam = U.CCLambda(cc, U.HBAR(H, cc))
    lam.compute_lambda()
    lref = O.CCLambda(ref, O.HBAR(ref.H, ref))
    lref.compute_lambda()
    assert np.abs(lam.l2 - lref.l2).max() < 2e-9


# members of one batch record the same operations: those without pairs on a side among themselves
@pytest.mark.parametrize("sizes", [[(1, 5), (1, 33)], [(2, 1), (3, 1)], SIZES[4:] + [(7, 40), (4, 96)]])
def test_batch_of_edge_sizes_matches_single_solves(sizes):
    hams = [make_hamiltonian(no, nv, 60 + k) for k, (no, nv) in enumerate(sizes)]
    bt = U.Batch()
    for h in hams:
        bt.add(h)
    e, _, ok = bt.ccsd({"R_CONVERGENCE": 1e-9})
    assert ok.all()
    for k, h in enumerate(hams):
        cc = U.CCWfn(U.Hamiltonian.from_synthetic(h), {"R_CONVERGENCE": 1e-9})
        cc.compute_energy()
        assert abs(cc.eccsd - e[k]) < 1e-10
        assert np.abs(bt.t2(k) - cc.t2).max() < 2e-9
