"""The byte-wise cost kernel of axis-aligned grey pairs of one focal length (layers of 16 M planes and pixels or more): raw
costs bit for bit against the oracle."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

THREADS = os.cpu_count() or 1


@pytest.fixture(scope="module")
def ctx():
    from lux_b200 import api
    c = api.Context(0)
    yield c
    c.close()


# widths below, at and past the 120-pixel runs and 128-pixel words, odd heights, a plane count that is no multiple of 32;
# the other camera's centre off by whole, half and quarter pixels (rounding tips single positions of a plane between two
# shifts) and outside the image for most planes; planes half a pixel apart; skipped pixels
@pytest.mark.parametrize("w,h,d,dcx,dcy,density,skip", [
    (720, 401, 64, 0.0, 0.0, 1.0, 0), (721, 333, 72, 0.5, 0.0, 1.0, 0), (839, 281, 80, 1.25, 0.0, 1.0, 2),
    (600, 500, 64, 0.25, 0.25, 1.0, 0), (607, 401, 72, -3.75, 0.5, 1.0, 2), (361, 600, 88, 40.0, -7.25, 1.0, 0),
    (961, 420, 48, 0.1, 0.0, 2.0, 0), (480, 700, 56, 470.0, 2.0, 1.0, 0)])
def test_unit_cost_bit_exact(ctx, oracle, w, h, d, dcx, dcy, density, skip):
    from lux_b200 import api, synth
    wl = synth.rectified_pair(w, h, d, seed=w + d, tile=16)
    f = np.float32(1000.0)
    cal = list(wl.calibs)
    cal[1] = api.CalibData(np.array([f, 0, w / 2.0 + dcx, 0, f, h / 2.0 + dcy, 0, 0, 1], np.float32), cal[1].T, cal[1].R)
    p = api.StereoParams(scale=1, tile=16, skip_mode=skip, plane_density=density)
    filt = [oracle.box_filter3(im) for im in wl.images]
    ol = oracle.layer(filt, wl.gray, cal, wl.near, wl.far, p, threads=THREADS)
    assert w * h * ol["n_planes"] >= 16 << 20
    gl = api.DenseLayer.compute(filt, wl.gray, cal, wl.near, wl.far, p, ctx=ctx)
    try:
        assert gl.cost_kernel == 3
        assert np.array_equal(gl.Skip.reshape(-1), ol["Skip"].reshape(-1))
        keep = np.repeat(ol["Skip"].reshape(-1) == 0, ol["n_planes"])
        assert np.array_equal(gl.Raw[keep], ol["Raw"][keep])
        assert not gl.Raw[~keep].any()
        assert np.array_equal(gl.Depth.view(np.uint32), ol["Depth"].view(np.uint32))
    finally:
        gl.close()


# its other size rule, 1184 tiles of 120 pixels and two rows: the smallest layers on either side of it, whole and quarter shifts
# with skipped pixels in layers past it
@pytest.mark.parametrize("w,h,d,dcx,dcy,density,skip", [
    (960, 296, 64, 0.0, 0.0, 1.0, 0), (959, 294, 64, 0.0, 0.0, 1.0, 0), (721, 401, 72, 0.5, 0.0, 1.0, 0), (839, 401, 80, 1.25, 0.0, 1.0, 2),
    (121, 1200, 128, -0.75, 0.0, 1.0, 0)])
def test_unit_cost_tile_rule(ctx, oracle, w, h, d, dcx, dcy, density, skip):
    test_unit_cost_bit_exact(ctx, oracle, w, h, d, dcx, dcy, density, skip)
