"""The census mode's paths along single lines against the oracle, bit for bit: the narrowest images they take and the widths below,
which walk scanlines; sides shorter than a segment; disparity ranges around the octets and lane widths; lines of a warp
that end one step apart; the largest penalties, one above the other; and a memory budget without room for the kept states."""
import numpy as np
import pytest

from oracle import census_oracle as C


def _images(w, h, seed):
    rng = np.random.default_rng(seed)
    left = rng.integers(0, 256, (h, w), dtype=np.uint8)
    right = np.roll(left, -2, axis=1)
    right[:: 3] = rng.integers(0, 256, right[:: 3].shape, dtype=np.uint8)
    left[h // 2:, : w // 2] = right[h // 2:, : w // 2] = 90  # flat: ties everywhere
    return left, right


@pytest.mark.gpu
@pytest.mark.parametrize("w,h,D,p1,p2", [
    (1, 1, 4, 10, 120), (7, 9, 16, 10, 120), (8, 1, 1, 10, 120), (8, 40, 33, 10, 120), (9, 3, 9, 10, 120), (40, 8, 255, 10, 120),
    (17, 16, 31, 10, 120), (27, 17, 128, 10, 120), (33, 25, 60, 10, 120), (31, 33, 8, 8129, 8129), (64, 9, 65, 8129, 7), (129, 41, 129, 0, 0),
    (200, 24, 24, 10, 120), (21, 90, 100, 10, 120)])
def test_lines_match_oracle(w, h, D, p1, p2):
    from lux_b200 import api
    left, right = _images(w, h, w * 7 + h)
    want = C.census_sgm(left, right, D, p1, p2)
    assert np.array_equal(api.CensusStereo.compute(left, right, D, p1, p2).view(np.uint32), want.view(np.uint32))
    want = C.census_sgm(left, right, D, p1, p2, lr_check=False)
    assert np.array_equal(api.CensusStereo.compute(left, right, D, p1, p2, lr_check=False).view(np.uint32), want.view(np.uint32))


@pytest.mark.gpu
def test_without_room_for_states():
    from lux_b200 import api
    w, h, D = 120, 64, 64
    left, right = _images(w, h, 3)
    need = 2 * w * h * 4 + w * h * (2 * 8 + 3 * D + 3 * 4) + 16 * 256  # images, censuses, costs, sums, disparities
    ctx = api.Context(0, hbm_budget_bytes=need)
    try:
        got = api.CensusStereo.compute(left, right, D, ctx=ctx)
    finally:
        ctx.close()
    assert np.array_equal(got.view(np.uint32), C.census_sgm(left, right, D, 10, 120).view(np.uint32))


@pytest.mark.gpu
@pytest.mark.parametrize("w,h,D", [(10, 30, 64), (10, 31, 64), (10, 31, 65), (8, 640, 70), (8, 641, 70), (8, 641, 16)])
def test_either_side_of_the_shape_rule(w, h, D):
    from lux_b200 import api
    left, right = _images(w, h, w + h)
    for lr in (True, False):
        want = C.census_sgm(left, right, D, 10, 120, lr_check=lr)
        assert np.array_equal(api.CensusStereo.compute(left, right, D, 10, 120, lr_check=lr).view(np.uint32), want.view(np.uint32))


@pytest.mark.gpu
def test_pairs_of_both_kinds_in_one_batch():
    """A tall image: pairs of up to 64 disparities walk scanlines, wider ones the lines, in the same batch."""
    from lux_b200 import api
    w, h, ds = 20, 100, [32, 100, 60, 200]
    pairs = [_images(w, h, 5 + k) for k in range(len(ds))]
    ref = pairs[0][0]
    others = [p[1] for p in pairs]
    _, disps = api.CensusStereo.capture(ref, others, ds, [1000.0] * len(ds))
    for k, d in enumerate(ds):
        assert np.array_equal(disps[k].view(np.uint32), C.census_sgm(ref, others[k], d, 10, 120).view(np.uint32)), k
