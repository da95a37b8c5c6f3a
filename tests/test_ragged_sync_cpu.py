"""Where the warps of lux_b200/csrc/sgm_ragged.cu must wait for their lanes: a model of which u16 of the two state copies
each lane reads and writes between two __syncwarp(). A lane of ragged_step and state_init holds aligned quads of the block's
planes; a lane of ragged_add takes four planes from the pixel's own first one on, which lie in other lanes' quads. Lanes may
run apart between two synchronisations (a lane past the pixel's planes leaves ragged_add early), so no two lanes may touch
a u16 there, one of them writing."""
import itertools

import pytest

LANES = 32


def _quads(copy, j0, j1, mode):
    """Every lane's own quads of rounds j0..j1."""
    return [(lane, (copy, 128 * j + 4 * lane + k), mode) for j in range(j0, j1 + 1) for lane in range(LANES) for k in range(4)]


class Warp:
    """The accesses of a warp's calls, cut into phases at each synchronisation."""

    def __init__(self, synced):
        self.synced, self.cur, self.phases = synced, 0, [[]]
        self.lo, self.hi = 1, 0

    def sync(self):
        self.phases.append([])

    def step(self, q, cap):
        j0, j1 = q // 128, (q + cap - 1) // 128
        own = _quads(self.cur, j0, j1, "r")
        beside = [(lane, (c, e + d), "r") for lane, (c, e), _ in own for d in ((-2, -1) if e % 4 == 0 else (1, 2) if e % 4 == 3 else ())]
        self.phases[-1] += own + beside + _quads(1 - self.cur, j0, j1, "w")
        self.flip()
        self.lo, self.hi = j0, j1
        self.sync()

    def add(self, q, cap):
        for w in range(cap // 4):
            first = q // 2 * 2 + 4 * w
            self.phases[-1] += [(w % LANES, (self.cur, first + k), "r") for k in range(6)]

    def init(self):
        if self.synced:
            self.sync()
        self.phases[-1] += _quads(self.cur, self.lo, self.hi, "w")
        self.lo, self.hi = 1, 0
        self.sync()

    def flip(self):
        self.cur = 1 - self.cur

    def revisit(self, odd):  # a band's first revisit in ragged_chain
        if odd:
            if self.synced:
                self.sync()
            self.flip()
        else:
            self.init()

    def conflicts(self):
        bad = 0
        for ph in self.phases:
            by = {}
            for lane, at, mode in ph:
                r, w = by.setdefault(at, (set(), set()))
                (w if mode == "w" else r).add(lane)
            bad += sum(len(w) > 1 or (len(w) == 1 and bool(r - w)) for r, w in by.values())
        return bad


RANGES = [(0, 64), (5, 56), (100, 40), (126, 8), (3, 200), (130, 120)]


def _walk(synced, between):
    warp = Warp(synced)
    for (q, cap), (q2, cap2) in itertools.product(RANGES, RANGES):
        warp.step(q, cap)
        warp.add(q, cap)
        between(warp)
        warp.step(q2, cap2)
        warp.add(q2, cap2)
    return warp.conflicts()


@pytest.mark.parametrize("between", [lambda w: None, lambda w: w.init(), lambda w: w.revisit(True), lambda w: w.revisit(False)],
                         ids=["the next pixel", "a new line", "an odd revisit", "a first revisit"])
def test_no_lane_overtakes_another(between):
    assert _walk(True, between) == 0


def test_the_synchronisations_are_needed():
    assert _walk(False, lambda w: None) == 0  # a step ends with one
    assert _walk(False, lambda w: w.init()) > 0
    assert _walk(False, lambda w: w.revisit(True)) > 0
