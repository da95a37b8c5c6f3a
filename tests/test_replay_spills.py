"""The exact replay on layers whose ranges reach past the last plane near pixels at the first planes: aggregates and depth bit for
bit against the oracle, on every solve. Such a pixel reads a few elements of the slot after its neighbour's, so the result
depends on where the row above stands (tests/test_replay_spills_cpu.py)."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

REPLAY = 0
THREADS = os.cpu_count() or 1


@pytest.fixture(scope="module")
def ctx():
    from lux_b200 import api
    c = api.Context(0)
    yield c
    c.close()


def test_pyramid_with_spills(ctx, oracle):
    from lux_b200 import api, synth
    cap = synth.capture(416, 312, 3, seed=5, f=332.8)
    ol = oracle.pyramid(cap.images, cap.gray, cap.calibs, cap.near, cap.far, threads=THREADS)
    for _ in range(3):
        gls = api.DenseStereoPyramid.run(cap.images, cap.gray, cap.calibs, cap.near, cap.far, keep_agg=True, ctx=ctx)
        try:
            assert any(g.sgm_kernel == REPLAY for g in gls[1:])
            for i in range(6):
                assert np.array_equal(gls[i].Agg, ol[i]["Agg"]), i
                assert np.array_equal(gls[i].Depth.view(np.uint32), ol[i]["Depth"].view(np.uint32)), i
        finally:
            for g in gls:
                g.close()


# parts of one, two, three and eight rows, a shorter last part, one band and several, a tile past the flag rows, an odd tile
@pytest.mark.parametrize("w,h,level,tile", [(400, 300, 4, 64), (402, 298, 4, 2), (330, 262, 4, 4), (300, 220, 4, 6), (516, 388, 4, 16),
                                            (330, 262, 5, 34), (264, 1040, 5, 32), (300, 220, 4, 128), (200, 150, 4, 5)])
@pytest.mark.parametrize("size", [1, 4])
def test_blocks_at_both_ends(ctx, oracle, w, h, level, tile, size):
    from lux_b200 import api, synth
    cap = synth.capture(w, h, 2, seed=w + level, f=0.8 * w)
    filt = [oracle.box_filter3(im) for im in cap.images]
    p = api.StereoParams.l16_pyramid()[level]
    p.tile = tile
    far = 640000.0
    planes = oracle.planes(cap.near, far, cap.calibs, p.plane_density, 8)
    n, pw, ph = len(planes), (w + 2 * p.scale - 1) // (2 * p.scale), (h + 2 * p.scale - 1) // (2 * p.scale)
    rng = np.random.default_rng(w * 10 + size)
    ends = np.concatenate([np.arange(4), np.arange(n - 6, n), [n // 2]])
    idx = np.kron(rng.choice(ends, (ph // size + 1, pw // size + 1)), np.ones((size, size), np.int64))[:ph, :pw]
    depth = planes[idx].astype(np.float32)
    ol = oracle.layer(filt, cap.gray, cap.calibs, cap.near, far, p, index=level, threads=1,
                      prev={"W": pw, "H": ph, "Depth": depth, "Skip": np.zeros((ph, pw), np.uint8)})
    assert ((ol["Start"].astype(int) - ol["MinLo"] + ol["Cap"]) > ol["MaxHi"] + 1).any()
    prev = api.DenseLayer.from_depth(depth, ctx=ctx)
    try:
        for _ in range(3):
            gl = api.DenseLayer.compute(filt, cap.gray, cap.calibs, cap.near, far, p, index=level, prev=prev, ctx=ctx)
            try:
                assert gl.sgm_kernel == REPLAY
                assert np.array_equal(gl.Agg, ol["Agg"])
                assert np.array_equal(gl.Depth.view(np.uint32), ol["Depth"].view(np.uint32))
            finally:
                gl.close()
    finally:
        prev.close()
