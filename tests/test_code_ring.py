"""The tensor-core GEMM's shared-memory and tensor-memory rings, as a model on the host: what its warps wait for and signal, with
copies and MMAs that complete in any order.  Checked are that a warp never reads a place before its copy has landed or after it was
asked for again, that no barrier gets an arrival its round has no room for, and that every warp comes to its end.

The model follows one pair of CTAs.  Where the packed codes go, and which barrier and parity a wait for them names, is the
library's own rule (nf4_prefill_code_place)."""
import ctypes
import random

import pytest

from unifur_b200 import _lib

BAR_RING = 8      # steps whose Full and Done barriers are told apart
COLUMN_SLOTS = 4  # steps of dequantised weights in tensor memory
WARPS = 16        # of a CTA that dequantise: four groups of four, two groups to a step


class Fault(Exception):
    pass


class Barrier:
    """An mbarrier: rounds of `count` arrivals and the bytes announced with them (in copies)."""

    def __init__(self, count):
        self.count, self.pending, self.copies, self.rounds = count, count, 0, 0

    def _turn(self):
        if self.pending == 0 and self.copies == 0:
            self.rounds += 1
            self.pending = self.count

    def arrive(self, copies=0):
        if self.pending == 0:
            raise Fault("an arrival that the barrier's round has no room for")
        self.pending -= 1
        self.copies += copies
        self._turn()

    def landed(self):
        self.copies -= 1
        self._turn()

    def passes(self, parity):  # try_wait.parity: the round of this parity is over
        return (self.rounds & 1) != parity


class Pair:
    def __init__(self, segments, x_slots, place, seed):
        """segments: (main k-stages, chunks of the adapter behind them) each; place(block) -> slot, barrier, parity."""
        self.rng, self.x_slots, self.place = random.Random(seed), x_slots, place
        # the steps of all segments: (block or None, stages)
        self.steps = []
        blocks = 0
        for stages, chunks in segments:
            for s in range(0, stages, 2):
                self.steps.append((blocks, min(2, stages - s)))
                blocks += 1
            self.steps += [(None, 0)] * chunks
        self.blocks = blocks
        places = [place(b) for b in range(64)]
        self.code_slots = max(p[0] for p in places) + 1
        n_full = max(p[1] for p in places) + 1
        self.full = [Barrier(1 + WARPS) for _ in range(BAR_RING)]                 # in the even CTA
        self.done = [[Barrier(1) for _ in range(BAR_RING)] for _ in range(2)]
        self.c_full = [[Barrier(1) for _ in range(n_full)] for _ in range(2)]
        self.c_empty = [[Barrier(8) for _ in range(self.code_slots)] for _ in range(2)]
        self.holds = [[None] * self.code_slots for _ in range(2)]                 # block whose codes have landed in a slot
        self.reading = [[0] * self.code_slots for _ in range(2)]                  # warps that still use them
        self.expanded = [0] * len(self.steps)                                     # warps that have, of a step
        self.x_landed = [0] * len(self.steps)
        self.mma_over = [False] * len(self.steps)
        self.flights = []                                                         # what may complete, in any order

    # every role is a generator: it yields a condition to wait for, and acts when that holds
    def code_warp(self, cta):
        for b in range(self.blocks):
            slot, bar, _ = self.place(b)
            yield lambda: self.c_empty[cta][slot].passes((b // self.code_slots & 1) ^ 1)
            if self.reading[cta][slot]:
                raise Fault(f"block {b} is asked for while its slot is read")
            self.c_full[cta][bar].arrive(copies=1)
            self.holds[cta][slot] = None

            def land(b=b, slot=slot, bar=bar):
                if self.reading[cta][slot]:
                    raise Fault(f"block {b} lands while its slot is read")
                self.holds[cta][slot] = b
                self.c_full[cta][bar].landed()

            self.flights.append(land)

    def producer(self, cta):
        user, slot = [None] * self.x_slots, 0
        for s, (block, _) in enumerate(self.steps):
            for _ in range(1 if block is not None else 2):
                last = user[slot]
                if last is not None:
                    yield lambda: self.done[cta][last % BAR_RING].passes(last // BAR_RING & 1)
                    if not self.mma_over[last]:
                        raise Fault(f"step {s} takes the place of step {last}, whose MMAs are under way")
                user[slot] = s
                slot = (slot + 1) % self.x_slots
            if cta == 0:
                self.full[s % BAR_RING].arrive(copies=2)

            def land(s=s):
                self.x_landed[s] += 1
                self.full[s % BAR_RING].landed()

            self.flights.append(land)

    def dequantiser(self, cta, warp):
        odd, half = warp >> 3, warp >> 2 & 1
        for s, (block, stages) in enumerate(self.steps):
            if s & 1 != odd:
                continue
            if block is not None:
                slot, bar, parity = self.place(block)
                yield lambda: self.c_full[cta][bar].passes(parity)
                if half < stages:
                    if self.holds[cta][slot] != block:
                        raise Fault(f"block {block} is read before it has landed")
                    self.reading[cta][slot] += 1
                else:
                    self.c_empty[cta][slot].arrive()
            yield lambda: s < COLUMN_SLOTS or self.done[cta][(s - COLUMN_SLOTS) % BAR_RING].passes((s - COLUMN_SLOTS) // BAR_RING & 1)
            if s >= COLUMN_SLOTS and not self.mma_over[s - COLUMN_SLOTS]:
                raise Fault(f"step {s} takes the columns of step {s - COLUMN_SLOTS}, whose MMAs are under way")
            self.expanded[s] += 1
            self.full[s % BAR_RING].arrive()
            if block is not None and half < stages:
                if self.holds[cta][slot] != block:
                    raise Fault(f"block {block} was overwritten while it was read")
                self.reading[cta][slot] -= 1
                self.c_empty[cta][slot].arrive()

    def issuer(self):
        for s in range(len(self.steps)):
            yield lambda: self.full[s % BAR_RING].passes(s // BAR_RING & 1)
            if self.expanded[s] != WARPS or self.x_landed[s] != 2:
                raise Fault(f"step {s} is multiplied before it is complete")

            def over(s=s):
                self.mma_over[s] = True
                for cta in range(2):
                    self.done[cta][s % BAR_RING].arrive()

            yield lambda: s == 0 or self.mma_over[s - 1]  # (MMAs complete in order)
            self.flights.append(over)

    def run(self):
        roles = [self.issuer()] + [r(c) for c in range(2) for r in (self.code_warp, self.producer)]
        roles += [self.dequantiser(c, w) for c in range(2) for w in range(WARPS)]
        waits = {i: None for i in range(len(roles))}
        for i in list(waits):
            self._next(roles, waits, i)
        # some runs let copies hang back, some let a CTA's or a pair of groups' warps run ahead
        lag = self.rng.choice((0.02, 0.2, 0.6))
        weight = {i: self.rng.choice((1, 1, 8)) for i in waits}
        while waits or self.flights:
            if self.flights and (self.rng.random() < lag or not self._ready(waits)):
                self.flights.pop(self.rng.randrange(len(self.flights)))()
                continue
            ready = self._ready(waits)
            if not ready:
                raise Fault("nobody can go on")
            self._next(roles, waits, self.rng.choices(ready, [weight[i] for i in ready])[0])

    @staticmethod
    def _ready(waits):
        return [i for i, w in waits.items() if w()]

    @staticmethod
    def _next(roles, waits, i):
        try:
            waits[i] = next(roles[i])
        except StopIteration:
            del waits[i]


SEGMENTS = [
    [(1, 0)], [(1, 1)], [(33, 1)], [(64, 0)], [(40, 3)],
    [(24, 1), (24, 1), (24, 1)],          # an odd number of chunks: the groups change sides against the slots
    [(7, 1), (9, 3), (5, 2), (1, 1), (13, 0), (3, 1)],  # odd last steps
    [(2, 1)] * 9, [(1, 0)] * 9, [(1, 4), (2, 1), (31, 1)],
    [(22, 0), (16, 2), (16, 2)],
]


def library_place(block):
    out = (ctypes.c_uint32 * 3)()
    assert _lib.load().nf4_prefill_code_place(block, out) >= 2
    return tuple(out)


@pytest.mark.parametrize("x_slots", [3, 6])  # wide and narrow tiles
@pytest.mark.parametrize("segments", SEGMENTS, ids=str)
def test_rings(segments, x_slots):
    for seed in range(12):
        Pair(segments, x_slots, library_place, seed).run()


@pytest.mark.parametrize("segments", [[(64, 0)], [(24, 1), (24, 1), (24, 1)]], ids=str)
def test_the_model_sees_a_wait_on_the_wrong_round(segments):
    # three slots with a barrier each, of which a pair of groups sees every second round
    def one_barrier_a_slot(block):
        return block % 3, block % 3, block // 3 & 1

    seen = set()
    for seed in range(40):
        try:
            Pair(segments, 6, one_barrier_a_slot, seed).run()
        except Fault as f:
            seen.add(" ".join(w for w in str(f).split() if not w.isdigit()))
    assert "block is read before it has landed" in seen


def test_places_are_a_ring():
    n = _lib.load().nf4_prefill_code_place(0, (ctypes.c_uint32 * 3)())
    places = [library_place(b) for b in range(8 * n)]
    for b, (slot, bar, parity) in enumerate(places):
        assert slot == b % n
        rounds = [i for i in range(b) if places[i][1] == bar]  # this barrier's earlier blocks
        assert parity == len(rounds) % 2 and all(places[i][0] == slot for i in rounds)
        # the one before has landed: the six steps' MMAs that a warp knows of at its turn for b
        assert not rounds or rounds[-1] <= b - 6
