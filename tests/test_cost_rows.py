"""The cost of uniform layers of several cameras (or of one that is not axis-aligned), eight planes a camera at a time: raw costs
bit for bit against the oracle."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _turn(R, deg, axis):
    c, s = np.cos(np.radians(deg)), np.sin(np.radians(deg))
    M = np.eye(3)
    i, j = [(1, 2), (0, 2), (0, 1)][axis]
    M[i, i], M[i, j], M[j, i], M[j, j] = c, -s, s, c
    return (M @ np.asarray(R, np.float64).reshape(3, 3)).astype(np.float32).reshape(np.asarray(R).shape)


# one warp's pixels and one past them, lone columns, one to many cameras, grey and colour, cameras turned so that the targets
# leave the rect and come back, or all lie outside it for whole groups of planes; skipped pixels; the layer scaled down
@pytest.mark.parametrize("w,h,n_cams,colour,deg,skip,scale", [
    (96, 40, 2, False, 0.5, 0, 1), (97, 33, 3, True, 1.5, 0, 1), (64, 31, 6, False, 4.0, 2, 1), (33, 50, 11, False, 1.0, 0, 1),
    (65, 24, 11, True, 6.0, 2, 1), (16, 8, 4, False, 0.2, 0, 1), (130, 66, 5, True, 2.0, 0, 2), (130, 66, 16, False, 2.0, 2, 2)])
def test_cost_rows_bit_exact(oracle, w, h, n_cams, colour, deg, skip, scale):
    from lux_b200 import api, synth
    cap = synth.capture(w, h, n_cams, seed=w + n_cams, f=0.75 * w, baseline_mm=(15.0, 50.0), colour=colour)
    cal = [api.CalibData(c.K, c.T, c.R if k == 0 else _turn(c.R, deg * (1 if k % 2 else -0.5), k % 3)) for k, c in enumerate(cap.calibs)]
    p = api.StereoParams(scale=scale, tile=8, skip_mode=skip, plane_density=1.0)
    filt = [oracle.box_filter3(im) for im in cap.images]
    ol = oracle.layer(filt, cap.gray, cal, cap.near, cap.far, p, threads=os.cpu_count() or 1)
    gl = api.DenseLayer.compute(filt, cap.gray, cal, cap.near, cap.far, p)
    try:
        assert gl.cost_kernel == 1
        keep = np.repeat(ol["Skip"].reshape(-1) == 0, ol["n_planes"])
        assert np.array_equal(gl.Raw[keep], ol["Raw"][keep])
        assert not gl.Raw[~keep].any()
    finally:
        gl.close()
