"""The ring of raw costs in column_chain (lux_b200/csrc/sgm_lines.cu): a model of which lane copies and reads which byte of the
two batch buffers between two __syncwarp(). A lane reads its own K planes of a step, but copies eight bytes of any lane's."""
import pytest

BATCH, LANES = 8, 32


def _copies(b, n):
    """stage(): lane and byte of the buffer it writes, rows of n planes one after the other."""
    oct_, out = n // 8, []
    for c in range(BATCH * oct_):
        i, part = divmod(c, oct_)
        out += [(c % LANES, (b & 1, i, part * 8 + k), "w") for k in range(8)]
    return out


def _reads(b, n, K):
    return [(lane, (b & 1, i, lane * K + k), "r") for i in range(BATCH) for lane in range(n // K) for k in range(K)]


def _conflicts(n, K, synced, batches=5):
    phases = [_copies(0, n) + _copies(1, n)]
    for b in range(batches):
        phases.append(_reads(b, n, K))  # cp_async_wait and __syncwarp before
        if synced:
            phases.append([])
        phases[-1] += _copies(b + 2, n)
    bad = 0
    for ph in phases:
        by = {}
        for lane, at, mode in ph:
            r, w = by.setdefault(at, (set(), set()))
            (w if mode == "w" else r).add(lane)
        bad += sum(len(w) > 1 or (len(w) == 1 and bool(r - w)) for r, w in by.values())
    return bad


@pytest.mark.parametrize("n,K", [(8, 4), (32, 4), (120, 4), (128, 4), (136, 8), (256, 8)])
def test_a_batch_is_read_before_it_is_replaced(n, K):
    assert _conflicts(n, K, True) == 0
    assert (_conflicts(n, K, False) > 0) == (n // 8 != LANES)  # 256 planes: every lane copies what it reads
