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
