"""Loads in flight when the CTAs of a pair leave a tensor-core GEMM after a wait has run out (tc_gemm.cu,
pair_drain), on a model of the ring: loads of both CTAs complete on rank 0's full barriers."""
import itertools
import random

import pytest


class Barrier:
    """An mbarrier with one expected arrival and a transaction count."""

    def __init__(self):
        self.phase, self.pending, self.tx = 0, 1, 0

    def _check(self):
        if self.pending == 0 and self.tx == 0:
            self.phase, self.pending = self.phase + 1, 1

    def arrive_expect(self, n):
        self.tx += n
        self.pending -= 1
        self._check()

    def complete(self, n):
        self.tx -= n
        self._check()

    def passed(self, phase):  # a wait with the parity of `phase`
        return self.phase > phase


def _leave(nst, stages, drain, seed):
    """Producers that stopped after stages[rank] stages.  Returns the loads that no wait covers: still in flight when
    every wait of rank 0 has returned."""
    rng = random.Random(seed)
    full = [Barrier() for _ in range(nst)]
    flight = []  # (rank, stage)
    waits = []  # phases that rank 0 awaits, in order

    def land(k):
        rank, n = flight.pop(k)
        full[n % nst].complete(1)

    def wait(n):  # a bounded wait: loads land at random until it passes or nothing is in flight (its limit)
        while not full[n % nst].passed(n // nst) and flight:
            land(rng.randrange(len(flight)))

    both = min(stages)
    for n in range(max(stages)):
        if n >= nst:  # a stage is issued again only when its last products have read it
            if n - nst < both:
                wait(n - nst)
        for rank in rng.sample((0, 1), 2):
            if n < stages[rank]:
                flight.append((rank, n))
                if rank == 0:
                    full[n % nst].arrive_expect(2)
    for n in range(max(0, stages[0] - nst), stages[0]):
        wait(n)
    if drain:
        for n in range(stages[0], stages[1]):
            full[n % nst].arrive_expect(1)
            wait(n)
    return list(flight)


@pytest.mark.parametrize("nst", [2, 3, 4, 6])
def test_no_load_in_flight_after_an_error(nst):
    missed = 0
    for first, ahead in itertools.product(range(0, 3 * nst), range(-nst, nst + 1)):
        stages = (first, first + ahead)
        if stages[1] < 0:
            continue
        for seed in range(5):
            assert not _leave(nst, stages, True, seed), stages
            missed += bool(_leave(nst, stages, False, seed))
            if ahead == 0:  # no error: nothing to drain
                assert not _leave(nst, stages, False, seed)
    assert missed  # without the drain the peer's surplus stays in flight
