"""Solves on a device whose memory others hold."""
import pytest

import ugacc_gb300 as U
from ugacc_gb300.generator import make_hamiltonian

OUT_OF_MEMORY = 3
MB = 1 << 20


class Held:
    """All device memory but `leave` bytes, held by this process."""

    def __init__(self, leave):
        self.leave = leave

    def __enter__(self):
        import torch

        free, _ = torch.cuda.mem_get_info()
        self.block = torch.empty(free - self.leave, dtype=torch.uint8, device="cuda")

    def __exit__(self, *exc):
        import torch

        del self.block
        torch.cuda.empty_cache()


def _load(no, nv):
    h = make_hamiltonian(no, nv, seed=9)
    return U.Hamiltonian(h.no, h.nv, h.fock, B=h.B)


@pytest.mark.gpu
def test_a_solve_after_one_that_ran_out_of_memory():
    """The first of the two blocks of the packed integrals fits (8256 x 8512 doubles, 536 MiB), the second does not."""
    opt = {"R_CONVERGENCE": 1e-9}
    ref = U.CCWfn(_load(2, 128), opt)
    ref.compute_energy()
    ref.ctx.close()
    cc = U.CCWfn(_load(2, 128), opt)
    with Held(800 * MB):
        with pytest.raises(U.UccError) as err:
            cc.compute_energy()
        assert err.value.status == OUT_OF_MEMORY
    assert cc.compute_energy() == ref.eccsd and cc.iterations == ref.iterations


def _rows_packed(cc):
    """Whether the last solve had Zmbij from the ladder's products: their counters include it."""
    no, nv = cc.no, cc.nv
    flops = cc.ctx.stats()["ladder_flops"] / cc.iterations
    assert flops in (2.0 * no ** 2 * nv ** 4, 2.0 * no ** 2 * nv ** 4 + 2.0 * no ** 3 * nv ** 3)
    return flops > 2.0 * no ** 2 * nv ** 4


@pytest.mark.gpu
@pytest.mark.parametrize("precision,start", [("FP64", 1400), ("MIXED", 2400)])
def test_solve_where_only_the_ladder_operator_fits(precision, start):
    """no=12, nv=96: the ladder's packed integrals take 324 MiB, the (m, b) rows 81 MiB.  From memory for both down,
    in steps of less than the rows: solves without the rows follow, to the same energy."""
    opt = {"R_CONVERGENCE": 1e-9, "PRECISION": precision}
    ref = U.CCWfn(_load(12, 96), opt)
    ref.compute_energy()
    assert _rows_packed(ref)
    ref.ctx.close()
    rows = []
    for leave in range(start, 200, -70):
        cc = U.CCWfn(_load(12, 96), opt)
        with Held(leave * MB):
            try:
                e = cc.compute_energy()
            except U.UccError as err:
                assert err.status == OUT_OF_MEMORY
                break
        # FP64: the same sweeps, a sum in another order.  Mixed: a residual of 1e-9 is some 1e-9 of energy
        assert abs(e - ref.eccsd) < (1e-12 if precision == "FP64" else 1e-8)
        rows.append(_rows_packed(cc))
        cc.ctx.close()
    assert rows[0] is True and rows[-1] is False and rows == sorted(rows, reverse=True)


@pytest.mark.gpu
def test_later_stage_takes_the_memory_of_the_packed_operator():
    """HBAR in less and less memory, in steps of less than the ladder's packed integrals take (367 MiB): before it does
    not fit at all, it fits in their place, and the next solve packs them again, without the (m, b) rows."""
    no, nv = 6, 96
    H = _load(no, nv)
    cc = U.CCWfn(H, {"R_CONVERGENCE": 1e-9})
    e = cc.compute_energy()
    hbar = U.HBAR(H, cc)
    ref = {k: hbar.block(k) for k in hbar.SHAPES}
    H.ctx.close()
    given_back = []
    for leave in range(4000, 200, -100):
        H = _load(no, nv)
        cc = U.CCWfn(H, {"R_CONVERGENCE": 1e-9})
        cc.compute_energy()
        with Held(leave * MB):
            try:
                hbar = U.HBAR(H, cc)
            except U.UccError as err:
                assert err.status == OUT_OF_MEMORY
                break
        for k in hbar.SHAPES:
            assert (hbar.block(k) == ref[k]).all(), (leave, k)
        H.ctx.reset_stats()
        assert abs(cc.compute_energy() - e) < 1e-12
        given_back.append(not _rows_packed(cc))
        H.ctx.close()
    assert given_back[0] is False and given_back[-1] is True and given_back == sorted(given_back)


@pytest.mark.gpu
def test_batch_where_the_packed_operators_do_not_fit():
    """Members whose packed integrals (2 x 375 MiB) do not fit are solved by the plain contractions."""
    members = [make_hamiltonian(4, 96, seed=k) for k in (1, 2)]

    def solve(leave):
        b = U.Batch()
        for h in members:
            b.add(h)
        with Held(leave * MB):
            out = b.ccsd({"R_CONVERGENCE": 1e-9})
        return (*out, b.info()["grouped_ops"])

    e, it, conv, ops = solve(4000)
    for leave, plain in ((1400, False), (500, True)):
        f, jt, conw, n = solve(leave)
        assert conv.all() and conw.all() and (it == jt).all() and (n != ops) == plain
        assert abs(e - f).max() < 1e-12
