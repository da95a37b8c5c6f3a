"""The last column's chain of the lines form against the revisit schedule (which the oracle's trace proves): per T-row band
of nr rows the chain visits rows 0..v-1 (v = min(K, nr), K = T - (W-1) mod T), revisits them, visits the rest, each step
from the state the step before left, but a band's first revisit from the newest state of the line-buffer half it looks
into: the last visit's for even v, the state before that for odd v."""
import pytest

from lux_b200 import api

INIT, EDGE, VISIT, REVISIT = 0, 1, 2 + 2, 2 + 4  # kSrcInit, kSrcEdge, kSrcCs + 2 (N(c).p2), kSrcCs + 4 (R(c).p2)


def _chain(W, H, T, second):
    """(row, revisit?, source) in the chain's order; a source is (kind, row)."""
    K = T - (W - 1) % T
    boundary = (EDGE if second else INIT, 0)
    out, state, before = [], boundary, boundary
    for base in range(0, H, T):
        nr = min(T, H - base)
        v = min(K, nr)
        for o in range(nr + v):
            rev = v <= o < 2 * v
            row = base + (o if o < v else o - v)
            if o == v and v % 2:
                state = before if row + v - 2 >= 0 else boundary
            out.append((row, rev, state))
            before, state = state, (REVISIT if rev else VISIT, row)
    return out


@pytest.mark.parametrize("second", [False, True])
def test_chain_matches_schedule(second):
    for T in (2, 4, 6, 16, 64):
        for W in list(range(8, 8 + T)) + [T + 1, 2 * T + 1, 4160, 4161]:
            if W < 8:
                continue
            for H in (2, 3, T - 1, T, T + 1, T + 2, 3 * T - 1, 3 * T, 3 * T + 1, 3 * T + 3):
                if H < 2:
                    continue
                sched, _, (end_first, end_count) = api.revisit_schedule(W, H, T, second)
                order = []
                for y in range(H):  # the schedule's order: a row's revisits, then its visit
                    first, count = int(sched[y][1]), int(sched[y][2])
                    order += [(first + k, True) for k in range(count)] + [(y, False)]
                order += [(end_first + k, True) for k in range(end_count)]
                chain = _chain(W, H, T, second)
                assert [(r, rev) for r, rev, _ in chain] == order, (W, H, T)
                for row, rev, src in chain:
                    if rev:
                        e = int(sched[row][5])
                        assert (e >> 24, e & 0xFFFFFF) == src, (W, H, T, row)
                    elif row > 0:
                        assert src == (REVISIT if sched[row][0] & 1 else VISIT, row - 1), (W, H, T, row)
