"""Kernels of one stream that start before their predecessor's writes are flushed: solves of the smallest
problems, where every kernel is short, have the same bits each time, alone and beside other contexts."""
import threading

import numpy as np
import pytest

import ugacc_gb300 as U
from ugacc_gb300.generator import make_hamiltonian


def _solve(no, nv):
    h = make_hamiltonian(no, nv, seed=11 * no + nv)
    H = U.Hamiltonian(h.no, h.nv, h.fock, B=h.B)
    cc = U.CCWfn(H, {"R_CONVERGENCE": 1e-9})
    cc.compute_energy()
    lam = U.CCLambda(cc, U.HBAR(H, cc))
    lam.compute_lambda()
    return cc.eccsd, cc.triples(), cc.t2, lam.l2


@pytest.mark.gpu
@pytest.mark.parametrize("no,nv", [(1, 3), (3, 9), (5, 19), (4, 33)])
def test_chained_launches_repeat_bits(no, nv):
    ref = _solve(no, nv)
    out = [None] * 12

    def work(first):
        for k in range(first, 12, 4):
            out[k] = _solve(no, nv)

    work(0)
    threads = [threading.Thread(target=work, args=(k,)) for k in (1, 2, 3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for got in out:
        assert all(np.array_equal(a, b) for a, b in zip(ref, got))
