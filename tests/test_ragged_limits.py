"""What the exact replay refuses stays refused for layers that the lines would take: a ragged layer whose line buffer is past the
replay's 32-bit indexing."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("w", [310000, 312000])  # just below and past 2^31 - 2^16 elements
def test_line_buffer_limit(w):
    from lux_b200 import api, synth
    h = 12
    cap = synth.capture(310000, h, 2, seed=9, f=3950.0)
    images = [np.ascontiguousarray(np.resize(im, (h, w, 4))) for im in cap.images]
    p = api.StereoParams.l16_pyramid()[5]
    planes = api.DenseStereo.planes(cap.near, 640000.0, cap.calibs, p.plane_density, 8)
    n, pw, ph = len(planes), w // 2, h // 2
    idx = np.full((ph, pw), n // 2)
    idx[:, :pw // 4] = 1  # ranges at both ends of the planes: MaxHi is all of them
    idx[2:4, pw // 2:pw // 2 + 20] = n - 4
    ctx = api.Context(0)
    try:
        prev = api.DenseLayer.from_depth(np.asarray(planes)[idx].astype(np.float32), ctx=ctx)
        try:
            def solve():
                return api.DenseLayer.compute(images, cap.gray, cap.calibs, cap.near, 640000.0, p, index=5, prev=prev,
                                              prefilter=True, ctx=ctx)
            if w < 311000:
                gl = solve()
                assert gl.sgm_kernel == 4 and 2 * (w + 2) * (4 * gl.MaxHi + 5) <= 2 ** 31 - 1 - 65536
                gl.close()
            else:
                with pytest.raises(api.LuxError) as e:
                    solve()
                assert "line buffer" in str(e.value)
        finally:
            prev.close()
    finally:
        ctx.close()
