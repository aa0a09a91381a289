"""Host model of the halo exchange of the resident sweeps (csrc/resident2d.cuh).

CTAs of a cluster pass their edge rows on by copies that complete the transaction count of an mbarrier in the
neighbour, one mbarrier per side and step parity. The model runs the threads of every CTA (the strip that waits for
and sends each edge, and the service warp that arms the mbarriers and sends a piece of its own) under random
schedules with copies delayed at will, and checks what the kernel relies on: a copy lands in the phase it was counted
for, and whoever sees a phase complete has all its rows. Waits may also give up at any time: the rest of the cluster then
still ends, arms no mbarrier twice, reads no row that has not arrived, and no transaction count runs off.
"""

from __future__ import annotations

import random

import pytest


class Violation(Exception):
    pass


class Mbarrier:
    """Arrival count 1 and a transaction count; phases are numbered by the steps they stand for."""

    def __init__(self, first):
        self.phase, self.pending, self.tx = first, 1, 0

    def arm(self, n):
        if self.pending != 1:
            raise Violation("armed before the phase before completed")
        self.pending, self.tx = 0, self.tx + n
        self._turn()

    def complete(self, n, phase, gave_up):
        if phase != self.phase and not gave_up:
            raise Violation(f"a copy of phase {phase} landed in phase {self.phase}")
        self.tx -= n
        if self.tx < -2 * (PIECES + 1):
            raise Violation("the transaction count runs off")
        self._turn()

    def _turn(self):
        if self.pending == 0 and self.tx == 0:
            self.phase, self.pending = self.phase + 2, 1

    def done(self, phase):  # by parity, as mbarrier.try_wait sees it
        return (self.phase - phase) % 4 == 2


PIECES = 2  # copies that make up an edge row


class Cluster:
    def __init__(self, n_ctas, steps, service_waits, rng, give_up=0.0, mute=False):
        self.n, self.steps, self.service_waits, self.rng, self.give_up = n_ctas, steps, service_waits, rng, give_up
        self.gave_up = [mute and c == 0 for c in range(n_ctas)]  # a mute CTA has given up before its first step
        self.bars = [[[Mbarrier(2), Mbarrier(1)] for _ in range(2)] for _ in range(n_ctas)]
        self.flight = []  # copies under way: (cta, side, phase)
        self.landed = {}
        self.at_barrier = [0] * n_ctas

    def has(self, cta, side):
        return cta > 0 if side == 0 else cta + 1 < self.n

    def wait(self, cta, side, m):  # False: given up
        while m > 0 and not self.bars[cta][side][m & 1].done(m):
            if self.gave_up[cta] or self.rng.random() < self.give_up:
                self.gave_up[cta] = True
                return False
            yield False
        if m > 0 and self.landed.get((cta, side, m), 0) != PIECES + (side == 0):
            raise Violation(f"step {m} of CTA {cta} reads rows that have not arrived")
        return True

    def send(self, cta, side, m):  # from this CTA towards `side`: the neighbour receives it on its other side
        self.flight.append((cta - 1 if side == 0 else cta + 1, 1 - side, m + 1))

    def cta_barrier(self, cta, m):
        self.at_barrier[cta] += 1
        while self.at_barrier[cta] < 3 * (m + 1):
            yield False

    def strip(self, cta, side):
        alive = not self.gave_up[cta]
        for m in range(self.steps):
            if self.has(cta, side):
                alive = alive and (yield from self.wait(cta, side, m))
                if alive and m + 1 < self.steps:
                    for _ in range(PIECES):
                        self.send(cta, side, m)
                        yield True
            yield from self.cta_barrier(cta, m)

    def service(self, cta):
        alive = not self.gave_up[cta]
        for m in range(self.steps):
            last = m + 1 == self.steps
            arm = not last and not self.gave_up[cta]
            for side in range(2):
                if self.has(cta, side) and arm:
                    self.bars[cta][side][(m + 1) & 1].arm(PIECES + (side == 0))
                    yield True
            if self.has(cta, 1) and not last:
                if self.service_waits:
                    alive = alive and (yield from self.wait(cta, 1, m))
                if alive:
                    self.send(cta, 1, m)
                    yield True
            yield from self.cta_barrier(cta, m)

    def land(self, i):
        cta, side, phase = self.flight.pop(i)
        self.landed[cta, side, phase] = self.landed.get((cta, side, phase), 0) + 1
        self.bars[cta][side][phase & 1].complete(1, phase, self.gave_up[cta])

    def run(self):
        threads = [t for c in range(self.n) for t in (self.strip(c, 0), self.strip(c, 1), self.service(c))]
        eager = self.rng.random()  # how readily copies land in this run
        idle = 0
        while threads:
            if self.flight and (idle > 3 * len(threads) or self.rng.random() < eager ** 3):
                self.land(self.rng.randrange(len(self.flight)))
                idle = 0
                continue
            t = self.rng.choice(threads)
            try:
                idle = 0 if next(t) else idle + 1
            except StopIteration:
                threads.remove(t)
                idle = 0
            if idle > (200 * self.n if self.give_up == 0 else 10**6) and not self.flight:  # (a wait may yet give up)
                raise Violation("no thread can go on")
        while self.flight:
            self.land(0)


@pytest.mark.parametrize("n_ctas", [2, 3, 5])
def test_copies_land_in_the_phase_they_are_counted_for(n_ctas):
    for seed in range(400):
        Cluster(n_ctas, 7, True, random.Random(seed)).run()


def test_a_service_piece_sent_without_the_wait_lands_in_the_phase_before():
    """Why the service warp waits for the rows below at every step it sends its piece, samples or not."""
    with pytest.raises(Violation, match="landed in phase"):
        for seed in range(400):
            Cluster(3, 7, False, random.Random(seed)).run()


@pytest.mark.parametrize("n_ctas", [2, 3, 5])
def test_a_wait_that_gives_up_leaves_the_others_sound(n_ctas):
    given = 0
    for seed in range(600):
        rng = random.Random(seed)
        c = Cluster(n_ctas, 9, True, rng, give_up=rng.choice([0.0005, 0.005, 0.2]), mute=seed % 3 == 0)
        c.run()
        given += any(c.gave_up) and seed % 3 > 0
    assert given > 100
