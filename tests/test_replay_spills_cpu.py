"""The exact replay's waits on layers whose ranges reach past the last plane (lux_b200/csrc/sgm_emulate.cu), checked on the
CPU with the happens-before model of test_replay_schedule_cpu.py.

A pixel whose padded range passes the block (q + cap > MaxHi + 1) reads, past its path-3 window, up to the first planes of
path 0's block in the slot after the neighbour's: of the row above's pixel two columns on in pass +1. The reference has
visited that pixel before, except from the last offset of a tile, where it comes later. The replay therefore lets such
a pixel wait for one offset more of the row above, and holds the row above at its next tile's start until such a pixel
at the end of the tile before has run."""
import random

import pytest

import test_replay_schedule_cpu as model

_count = model._count_unordered


def _graph(W, H, T, dirn, high, ordered, monkeypatch):
    """Unordered pairs (or -1) of the replay's waits with the given high pixels (row, column of the pass); ordered: with the
    waits for them."""
    R = model.launcher_part_rows(T)
    parts = (T + R - 1) // R
    gwN = (W + 2 * T - 1) // T
    result = []

    def extended(ids, preds, pixels):
        key_of = {n: k for k, n in ids.items()}

        def edge(a, b):
            preds.setdefault(b, set()).add(ids[a])

        def band_rows(j):
            return min(T, H - j * T)
        out = []
        for ref, n, (w, rd) in pixels:
            j, part, r, i, u = key_of[n]
            xp = model._pixel_xp(W, T, i, r, u)
            hb = 0 if r % 2 == 0 else 1  # the other half of the line buffer
            if (j * T + r, xp) in high:
                past = xp + 2 if dirn > 0 else xp
                rd = rd | {(hb, "b0", past), (hb, "body", past)}
                if ordered and dirn > 0 and xp + 2 < W:
                    if r == 0 and j > 0:  # the band above comes first: its last row, one offset more
                        t = min((i + 1) * T + u + 2, gwN * T) - 1
                        edge((j - 1, parts - 1, T - 1, t // T, t % T), n)
                    elif r > 0 and u + 1 < T:
                        edge((j, (r - 1) // R, r - 1, i, u + 1), n)
            if ordered and dirn > 0 and u == 0 and i > 0 and r + 1 < band_rows(j) and i * T - r < W and xp >= 2 and (j * T + r + 1, xp - 2) in high:
                if (r + 1) // R == part:  # the row below has finished the tile before
                    edge((j, part, r + 1, i - 1, T - 1), n)
                else:  # the part below's last row has
                    below = min((part + 2) * R, band_rows(j)) - 1
                    edge((j, part + 1, below, i - 1, T - 1), n)
            out.append((ref, n, (w, rd)))
        result.append(_count(ids, preds, out))
        return 0

    monkeypatch.setattr(model, "_count_unordered", extended)
    model.unordered_pairs(W, H, T, 0, dirn, part_rows=R)
    return result[0]


def _everywhere(W, H):
    return {(y, x) for y in range(H) for x in range(W)}


SIZES = [(65, 49, 4), (48, 40, 8), (97, 61, 16), (70, 45, 32), (66, 65, 64), (33, 17, 2), (20, 11, 6), (75, 70, 34), (61, 55, 50)]


@pytest.mark.parametrize("W,H,T", SIZES)
@pytest.mark.parametrize("dirn", [1, -1])
def test_ordered_with_every_pixel_high(W, H, T, dirn, monkeypatch):
    assert _graph(W, H, T, dirn, _everywhere(W, H), True, monkeypatch) == 0


@pytest.mark.parametrize("W,H,T", SIZES)
def test_ordered_with_some_pixels_high(W, H, T, monkeypatch):
    rng = random.Random(W * H)
    high = set(rng.sample(sorted(_everywhere(W, H)), W * H // 10))
    assert _graph(W, H, T, 1, high, True, monkeypatch) == 0


@pytest.mark.parametrize("W,H,T", [(65, 49, 4), (70, 45, 32), (66, 65, 64)])
def test_the_plain_waits_leave_them_unordered(W, H, T, monkeypatch):
    """One pixel past the last plane, inside a tile or at its end, meets the row above unordered in pass +1."""
    for x in (T // 2, T - 2):  # row 1 of the first band: column iT - 1 + u
        high = {(1, x)}
        assert _graph(W, H, T, 1, high, False, monkeypatch) > 0
        assert _graph(W, H, T, 1, high, True, monkeypatch) == 0
        assert _graph(W, H, T, -1, high, False, monkeypatch) == 0
