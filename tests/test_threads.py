"""Layers of different sizes solved at once from several threads, a context each: what one launch asks of a kernel (its shared
memory above all) must not depend on another thread's layer. Every result equals the same layer solved alone."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _ragged(oracle, w, h, f, level):
    from lux_b200 import api, synth
    cap = synth.capture(w, h, 2, seed=w, f=f)
    filt = [oracle.box_filter3(im) for im in cap.images]
    p = api.StereoParams.l16_pyramid()[level]
    planes = oracle.planes(cap.near, 640000.0, cap.calibs, p.plane_density, 8)
    pw, ph = (w + 2 * p.scale - 1) // (2 * p.scale), (h + 2 * p.scale - 1) // (2 * p.scale)
    depth = planes[12 + np.random.default_rng(w).integers(0, len(planes) - 24, (ph, pw))].astype(np.float32)

    def solve(ctx):
        prev = api.DenseLayer.from_depth(depth, ctx=ctx)
        gl = api.DenseLayer.compute(filt, cap.gray, cap.calibs, cap.near, 640000.0, p, index=level, prev=prev, ctx=ctx)
        try:
            return gl.sgm_kernel, gl.MaxHi, gl.Depth.copy()
        finally:
            gl.close()
            prev.close()
    return solve


def _uniform(oracle, w, h, d, sgm):
    from lux_b200 import api, synth
    wl = synth.rectified_pair(w, h, d, seed=w + d, tile=16)
    filt = [oracle.box_filter3(im) for im in wl.images]

    def solve(ctx):
        gl = api.DenseLayer.compute(filt, wl.gray, wl.calibs, wl.near, wl.far, wl.params, sgm=sgm, ctx=ctx)
        try:
            return gl.sgm_kernel, gl.MaxHi, gl.Depth.copy()
        finally:
            gl.close()
    return solve


@pytest.mark.parametrize("kind", ["ragged", "chains"])
def test_concurrent_layers_equal_solo(oracle, kind):
    from lux_b200 import api
    if kind == "ragged":
        solves = [_ragged(oracle, 400, 300, 320.0, 4), _ragged(oracle, 400, 300, 2400.0, 4)]
    else:
        solves = [_uniform(oracle, 150, 100, d, "split") for d in (136, 256)]
    ctxs = [api.Context(0) for _ in solves]
    try:
        solo = [s(c) for s, c in zip(solves, ctxs)]
        assert solo[0][0] == solo[1][0] == (4 if kind == "ragged" else 2)
        assert solo[1][1] > 1.5 * solo[0][1]  # plane counts, and with them the shared memory
        errors = []

        def run(k):
            try:
                for _ in range(40):
                    form, _, depth = solves[k](ctxs[k])
                    if form != solo[k][0] or not np.array_equal(depth.view(np.uint32), solo[k][2].view(np.uint32)):
                        errors.append(f"layer {k} differs")
            except Exception as e:  # noqa: BLE001
                errors.append(repr(e))
        threads = [threading.Thread(target=run, args=(k,)) for k in range(2)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert not errors, errors[:3]
    finally:
        for c in ctxs:
            c.close()
