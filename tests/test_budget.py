"""Solves under an HBM budget that held them before the lines forms and the byte-wise cost: where the memory that those take is
not there, the solve runs without it, and the bits are the same."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LINES, FUSED, REPLAY = 4, 1, 0


def _bits(a):
    return a.view(np.uint32)


def _solve(wl, budget=0, autotune=True, **kw):
    """(form, cost kernel, depth, device bytes at the peak) of a solve in a context of its own."""
    from lux_b200 import api
    ctx = api.Context(0, hbm_budget_bytes=budget)
    try:
        ctx.set_autotune(autotune)
        api.pool_high_water(0, reset=True)
        base = api.pool_high_water(0)
        gl = api.DenseLayer.compute(wl.images, wl.gray, wl.calibs, wl.near, wl.far, wl.params, prefilter=True, ctx=ctx, **kw)
        try:
            return gl.sgm_kernel, gl.cost_kernel, gl.Depth.copy(), api.pool_high_water(0) - base
        finally:
            gl.close()
    finally:
        ctx.close()


def test_without_the_kept_states():
    """2080x1560 D=256: the lines' kept states are 0.43 GB; a budget that holds the fused form has no room for them."""
    from lux_b200 import synth
    wl = synth.rectified_pair(2080, 1560, 256, seed=21, bits=12, tile=64)
    form, _, depth, peak = _solve(wl)
    assert form == LINES
    form, _, fused, peak_fused = _solve(wl, sgm="fused")
    assert form == FUSED and np.array_equal(_bits(fused), _bits(depth))
    assert peak > peak_fused + (200 << 20)
    form, _, got, _ = _solve(wl, budget=peak_fused)
    assert form == LINES and np.array_equal(_bits(got), _bits(depth))


def test_without_the_lines_tables():
    """Eight planes and a tall, narrow layer: the lines' column states (for 256 planes) are larger than the fused form's."""
    from lux_b200 import synth
    wl = synth.rectified_pair(9, 60001, 8, seed=22, tile=8)
    form, _, depth, peak = _solve(wl)
    assert form == LINES
    form, _, fused, peak_fused = _solve(wl, sgm="fused")
    assert form == FUSED and np.array_equal(_bits(fused), _bits(depth))
    assert peak > peak_fused
    form, _, got, _ = _solve(wl, budget=peak_fused, autotune=False)
    assert form == FUSED and np.array_equal(_bits(got), _bits(depth))


def test_without_the_byte_phase_images():
    """A narrow pair past the byte-wise cost's size rule: its phase images have 512 bytes of padding a row (43 MB here; the
    triples 9 MB)."""
    from lux_b200 import synth
    wl = synth.rectified_pair(64, 4200, 64, seed=23, tile=64)
    _, kind, depth, peak = _solve(wl)
    assert kind == 3
    budget = 64 * 4200 * (3 * 64 + 23 + 16 + 32) + (12 << 20)
    assert peak > budget
    _, kind, got, _ = _solve(wl, budget=budget)
    assert kind == 3 and np.array_equal(_bits(got), _bits(depth))


def test_ragged_without_the_lines_tables(oracle):
    from lux_b200 import api, synth
    w, h = 2000, 40
    cap = synth.capture(w, h, 2, seed=9, f=330.0)
    filt = [oracle.box_filter3(im) for im in cap.images]
    p = api.StereoParams.l16_pyramid()[5]
    planes = oracle.planes(cap.near, 640000.0, cap.calibs, p.plane_density, 8)
    pw, ph = (w + 2 * p.scale - 1) // (2 * p.scale), (h + 2 * p.scale - 1) // (2 * p.scale)
    depth = planes[12 + np.random.default_rng(1).integers(0, len(planes) - 24, (ph, pw))].astype(np.float32)

    def solve(budget=0, **kw):
        ctx = api.Context(0, hbm_budget_bytes=budget)
        try:
            prev = api.DenseLayer.from_depth(depth, ctx=ctx)
            api.pool_high_water(0, reset=True)
            base = api.pool_high_water(0)
            gl = api.DenseLayer.compute(filt, cap.gray, cap.calibs, cap.near, 640000.0, p, index=5, prev=prev, ctx=ctx, **kw)
            try:
                return gl.sgm_kernel, gl.Agg.copy(), gl.Depth.copy(), api.pool_high_water(0) - base
            finally:
                gl.close()
                prev.close()
        finally:
            ctx.close()
    form, agg, d, peak = solve()
    assert form == LINES
    form, agg1, d1, peak_replay = solve(force_replay=True)
    assert form == REPLAY and np.array_equal(agg, agg1) and np.array_equal(_bits(d), _bits(d1))
    assert peak > peak_replay
    form, agg2, d2, _ = solve(budget=peak_replay + 2 * pw * ph * 5 + (1 << 16))  # (the depth map it continues from is counted too)
    assert form == REPLAY and np.array_equal(agg, agg2) and np.array_equal(_bits(d), _bits(d2))
