"""The lines form of the uniform aggregation (every path along its own lines, sgm_kernel 4), which a layer takes when pass
+1's aggregates are not kept: bit for bit against the oracle at the sizes where it can go wrong. Layers below its size rule
run a pass's paths at once; past it the checkpointed walks run, in segments of eight pixels."""
import os

import numpy as np
import pytest

from test_gpu_parity import UNIFORM_CASES

pytestmark = pytest.mark.gpu

LINES = 4


@pytest.fixture(scope="module")
def ctx():
    from lux_b200 import api
    c = api.Context(0)
    yield c
    c.close()


def _solve(ctx, wl, **kw):
    from lux_b200 import api
    gl = api.DenseLayer.compute(wl.images, wl.gray, wl.calibs, wl.near, wl.far, wl.params, prefilter=True, ctx=ctx, **kw)
    try:
        return gl.sgm_kernel, gl.Agg if kw.get("keep_agg") else None, gl.Depth
    finally:
        gl.close()


# the other forms' cases (lane widths, padding lanes, revisit counts, partial bands), then: eight columns, four rows, fewer
# steps than a batch, one plane octet, a full 32, 64 and 128 planes, every row revisited (T divides W - 1)
@pytest.mark.parametrize("w,h,d,tile", [c for c in UNIFORM_CASES if c[0] >= 8] + [(8, 4, 8, 2), (9, 7, 8, 4), (200, 4, 16, 8), (8, 150, 32, 64),
                                                        (65, 65, 64, 64), (129, 50, 128, 8), (97, 301, 248, 16)])
def test_lines_small_form_bit_exact(ctx, oracle, w, h, d, tile):
    from lux_b200 import synth
    wl = synth.rectified_pair(w, h, d, seed=w * 3 + h, tile=tile)
    filt = [oracle.box_filter3(im) for im in wl.images]
    ol = oracle.layer(filt, wl.gray, wl.calibs, wl.near, wl.far, wl.params)
    form, agg, depth = _solve(ctx, wl, keep_agg=True)
    assert form == LINES
    assert np.array_equal(agg, ol["Agg"])
    assert np.array_equal(depth.view(np.uint32), ol["Depth"].view(np.uint32))
    form, _, depth = _solve(ctx, wl)
    assert form == LINES and np.array_equal(depth.view(np.uint32), ol["Depth"].view(np.uint32))


@pytest.mark.parametrize("w,h,d,tile", [(1301, 1210, 176, 64), (2177, 1903, 64, 32)])
def test_lines_large_form_bit_exact(ctx, oracle, w, h, d, tile):
    from lux_b200 import synth
    wl = synth.rectified_pair(w, h, d, seed=7, tile=tile)
    filt = [oracle.box_filter3(im) for im in wl.images]
    ol = oracle.layer(filt, wl.gray, wl.calibs, wl.near, wl.far, wl.params, threads=os.cpu_count() or 1)
    form, agg, depth = _solve(ctx, wl, keep_agg=True)
    assert form == LINES
    assert np.array_equal(agg, ol["Agg"])
    assert np.array_equal(depth.view(np.uint32), ol["Depth"].view(np.uint32))


# segments that do not divide a side, one-segment sides, a line per warp / two / four, odd heights (pass -1 starts from the
# row above the last), tiles whose every row revisits the last column
@pytest.mark.parametrize("w,h,d,tile", [(1601, 801, 256, 64), (120001, 9, 256, 8), (3000, 703, 120, 16), (17, 62000, 256, 16),
                                        (4160, 650, 96, 64), (1283, 1527, 136, 2)])
def test_lines_large_form_equals_chains(ctx, w, h, d, tile):
    from lux_b200 import synth
    wl = synth.rectified_pair(w, h, d, seed=11, tile=tile)
    form, agg, depth = _solve(ctx, wl, keep_agg=True)
    assert form == LINES
    form, agg2, depth2 = _solve(ctx, wl, keep_agg=True, sgm="split")
    assert form == 2
    assert np.array_equal(agg, agg2)
    assert np.array_equal(depth.view(np.uint32), depth2.view(np.uint32))
    form, _, depth3 = _solve(ctx, wl)
    assert form == LINES and np.array_equal(depth3.view(np.uint32), depth2.view(np.uint32))


def test_lines_yields_to_pass1_and_chosen_forms(ctx):
    """Where pass +1's aggregates are kept, or the caller chose a form for the shape, the other forms run as before."""
    from lux_b200 import api, synth
    wl = synth.rectified_pair(123, 77, 40, seed=2, tile=16)
    assert _solve(ctx, wl)[0] == LINES
    assert _solve(ctx, wl, keep_pass1=True)[0] in (1, 2, 3)
    assert _solve(ctx, wl)[0] == LINES  # a timed choice is not the caller's
    try:
        api.set_tuned_form(123, 77, 40, 16, 3)
        assert _solve(ctx, wl)[0] == 3
    finally:
        api.set_tuned_form(123, 77, 40, 16, 0)
    assert _solve(ctx, wl)[0] == LINES


# the large form of four and two lines a warp, and the small form's widths of four planes a lane on either side of its limits
@pytest.mark.parametrize("w,h,d,tile", [(2901, 2803, 64, 32), (2101, 1903, 128, 64), (1999, 1901, 128, 64), (611, 333, 16, 64), (413, 301, 24, 32),
                                        (300, 211, 40, 16), (301, 203, 72, 64), (250, 120, 128, 8), (250, 120, 136, 8)])
def test_lines_lane_widths_equal_chains(ctx, w, h, d, tile):
    from lux_b200 import synth
    wl = synth.rectified_pair(w, h, d, seed=17, tile=tile)
    form, agg, depth = _solve(ctx, wl, keep_agg=True)
    assert form == LINES
    form, agg2, depth2 = _solve(ctx, wl, keep_agg=True, sgm="split")
    assert form == 2
    assert np.array_equal(agg, agg2)
    assert np.array_equal(depth.view(np.uint32), depth2.view(np.uint32))
    form, _, depth3 = _solve(ctx, wl)
    assert form == LINES and np.array_equal(depth3.view(np.uint32), depth2.view(np.uint32))
