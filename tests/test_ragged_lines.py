"""The lines form of ragged layers (sgm_kernel 4 where pass +1's aggregates are not kept): aggregates and depth bit for bit
against the oracle, on pyramids, on layers continued from depth maps made for the ends of the plane range, and on uniform
layers past 256 planes; and the layers that must keep the exact replay, because a range reaches past the last plane of the
reference's line-buffer block near one that starts at its first planes."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LINES, REPLAY = 4, 0
THREADS = os.cpu_count() or 1


@pytest.fixture(scope="module")
def ctx():
    from lux_b200 import api
    c = api.Context(0)
    yield c
    c.close()


def _same(gl, ol, tag):
    assert (gl.MinLo, gl.MaxHi) == (ol["MinLo"], ol["MaxHi"]), tag
    assert np.array_equal(gl.Agg, ol["Agg"]), tag
    assert np.array_equal(gl.Depth.view(np.uint32), ol["Depth"].view(np.uint32)), tag


def test_pyramid_without_pass1(ctx, oracle):
    from lux_b200 import api, synth
    cap = synth.capture(416, 312, 3, seed=5, f=330.0)
    ol = oracle.pyramid(cap.images, cap.gray, cap.calibs, cap.near, cap.far, threads=THREADS)
    gls = api.DenseStereoPyramid.run(cap.images, cap.gray, cap.calibs, cap.near, cap.far, keep_agg=True, ctx=ctx)
    try:
        assert sum(g.sgm_kernel == LINES for g in gls) >= 4
        for i in range(6):
            assert gls[i].sgm_kernel in (LINES, REPLAY)
            _same(gls[i], ol[i], f"L{i}")
    finally:
        for g in gls:
            g.close()


def _resume(ctx, oracle, w, h, level, depth_of, tile=None, cams=2, far=640000.0):
    """A layer continued from the depth map depth_of(planes, ph, pw) gives, on the GPU and the oracle."""
    from lux_b200 import api, synth
    cap = synth.capture(w, h, cams, seed=w + level, f=0.8 * w)
    filt = [oracle.box_filter3(im) for im in cap.images]
    p = api.StereoParams.l16_pyramid()[level]
    if tile:
        p.tile = tile
    planes = oracle.planes(cap.near, far, cap.calibs, p.plane_density, 8)
    pw, ph = (w + 2 * p.scale - 1) // (2 * p.scale), (h + 2 * p.scale - 1) // (2 * p.scale)
    depth = depth_of(planes, ph, pw).astype(np.float32)
    ol = oracle.layer(filt, cap.gray, cap.calibs, cap.near, far, p, index=level, threads=THREADS,
                      prev={"W": pw, "H": ph, "Depth": depth, "Skip": np.zeros((ph, pw), np.uint8)})
    prev = api.DenseLayer.from_depth(depth, ctx=ctx)
    gl = api.DenseLayer.compute(filt, cap.gray, cap.calibs, cap.near, far, p, index=level, prev=prev, ctx=ctx)
    try:
        if gl.sgm_kernel == LINES:
            _same(gl, ol, f"{w}x{h} level {level} tile {p.tile}")
        return gl.sgm_kernel, ol
    finally:
        gl.close()
        prev.close()


def _blocks(rng, n, ph, pw, size=5):
    """Plane indices constant over blocks of several pixels: ranges of every start and length."""
    b = rng.integers(0, n, (ph // size + 1, pw // size + 1))
    return np.kron(b, np.ones((size, size), np.int64))[:ph, :pw]


# every revisit count class (W - 1 mod tile), odd heights, one band and several, tiles of two rows
@pytest.mark.parametrize("w,h,level,tile", [(400, 300, 3, 32), (402, 298, 4, 64), (330, 262, 5, 64), (516, 388, 4, 2),
                                            (520, 260, 4, 128), (264, 1040, 5, 16)])
def test_resumed_layer(ctx, oracle, w, h, level, tile):
    rng = np.random.default_rng(w + tile)

    def depth(planes, ph, pw):  # away from both ends of the planes
        n = len(planes)
        return planes[12 + _blocks(rng, max(1, n - 40), ph, pw)]
    form, ol = _resume(ctx, oracle, w, h, level, depth, tile=tile)
    assert form == LINES
    assert len(np.unique(ol["Start"] % 4)) == 4 and ol["Cap"].min() < ol["Cap"].max()


def test_ranges_past_the_last_plane(ctx, oracle):
    """A patch of ranges whose padded end passes MaxHi, far from any range at the first planes: plain values, lines."""
    def depth(planes, ph, pw):
        n = len(planes)
        idx = np.full((ph, pw), n // 2)
        idx[ph // 4: ph // 2, pw // 4: pw // 2] = n - 3
        idx[3 * ph // 4:, : pw // 4] = 0  # the first planes, elsewhere
        return planes[idx]
    form, ol = _resume(ctx, oracle, 400, 300, 4, depth)
    assert ((ol["Start"].astype(int) - ol["MinLo"] + ol["Cap"]) > ol["MaxHi"] + 1).any()
    assert form == LINES


@pytest.mark.parametrize("where", ["beside the first planes", "at the border"])
def test_spills_keep_the_replay(ctx, oracle, where):
    def depth(planes, ph, pw):
        n = len(planes)
        idx = np.full((ph, pw), n // 2)
        idx[3 * ph // 4:, : pw // 4] = 0
        if where == "beside the first planes":
            idx[ph // 2: 3 * ph // 4, : pw // 4] = n - 3
        else:
            idx[: ph // 4, -3:] = n - 3
        return planes[idx]
    form, ol = _resume(ctx, oracle, 400, 300, 4, depth)
    assert ((ol["Start"].astype(int) - ol["MinLo"] + ol["Cap"]) > ol["MaxHi"]).any()
    assert form == REPLAY


@pytest.mark.parametrize("w,h,d,tile", [(600, 40, 264, 8), (520, 48, 400, 16), (700, 30, 552, 4), (300, 20, 768, 2)])
def test_wide_uniform_layer(ctx, oracle, w, h, d, tile):
    from lux_b200 import api, synth
    wl = synth.rectified_pair(w, h, d, seed=d + tile, tile=tile)
    filt = [oracle.box_filter3(im) for im in wl.images]
    ol = oracle.layer(filt, wl.gray, wl.calibs, wl.near, wl.far, wl.params)
    for keep in (True, False):
        gl = api.DenseLayer.compute(filt, wl.gray, wl.calibs, wl.near, wl.far, wl.params, keep_agg=keep, ctx=ctx)
        try:
            assert gl.sgm_kernel == LINES
            if keep:
                _same(gl, ol, f"{w}x{h} D{d}")
            assert np.array_equal(gl.Depth.view(np.uint32), ol["Depth"].view(np.uint32))
        finally:
            gl.close()
