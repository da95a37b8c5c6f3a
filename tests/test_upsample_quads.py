"""The upsample by quads of output pixels (four that share their low-resolution pixels) and the border pixel by pixel, against the
oracle bit for bit: sizes without quads, with one, around a block's 256 quads; with and without confidence; a guide at an odd address; exponents beyond the range that the weights clamp, and depths whose reciprocal is not a normal number."""
import ctypes

import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("pw,ph,gw,gh,with_conf,sigma", [
    (1, 1, 2, 2, True, 10.0), (2, 2, 4, 4, True, 10.0), (2, 9, 4, 18, False, 10.0), (3, 2, 6, 4, True, 0.5), (257, 2, 514, 4, False, 10.0),
    (17, 17, 34, 34, True, 1e-3), (16, 16, 32, 32, False, 300.0), (129, 31, 258, 62, True, 10.0)])
def test_quads(oracle, pw, ph, gw, gh, with_conf, sigma):
    from lux_b200 import api
    rng = np.random.default_rng(pw * 100 + ph)
    depth = rng.uniform(300.0, 6000.0, (ph, pw)).astype(np.float32)
    depth.reshape(-1)[::7] = [np.float32(v) for v in np.resize([0.0, -0.0, np.inf, 1e-40, 3e38, -5.0], depth.reshape(-1)[::7].size)]
    guide = rng.integers(0, 256, (gh, gw, 4), dtype=np.uint8)
    guide[: gh // 2] = 255  # flat: every weight's exponent is -0
    conf = rng.uniform(0, 1, (ph, pw)).astype(np.float32) if with_conf else None
    od, oc = oracle.upsample(depth, pw, ph, guide, pw, ph, sigma=sigma, prev_conf=conf)
    r = api.DenseUpsampleLayer.run(depth, pw, ph, guide, pw, ph, sigma=sigma, prev_confidence=conf)
    same = (r.Depth.reshape(od.shape).view(np.uint32) == od.view(np.uint32)) | (np.isnan(od) & np.isnan(r.Depth.reshape(od.shape)))
    assert same.all()
    if with_conf:
        assert np.array_equal(r.Confidence.reshape(oc.shape).view(np.uint32), oc.view(np.uint32))


@pytest.mark.gpu
def test_guide_at_an_odd_address(oracle):
    import torch
    from lux_b200 import _lib, api
    pw, ph = 33, 9
    rng = np.random.default_rng(5)
    depth = rng.uniform(300.0, 6000.0, (ph, pw)).astype(np.float32)
    guide = rng.integers(0, 256, (2 * ph, 2 * pw, 4), dtype=np.uint8)
    ctx = api.default_context()
    d_prev = torch.from_numpy(depth).cuda()
    d_guide = torch.zeros(guide.size + 16, dtype=torch.uint8, device="cuda")
    d_guide[1:1 + guide.size] = torch.from_numpy(guide.reshape(-1)).cuda()
    d_out = torch.zeros(2 * ph, 2 * pw, device="cuda")
    torch.cuda.synchronize()
    img = _lib.Img(d_guide.data_ptr() + 1, 2 * pw, 2 * ph, 2 * pw, 1)
    ctx.check(ctx.lib.lux_sgm_upsample_noalloc(ctx.handle, d_prev.data_ptr(), pw, ph, ctypes.byref(img), pw, ph, 12.0, 2, None,
                                               d_out.data_ptr(), None))
    od, _ = oracle.upsample(depth, pw, ph, guide, pw, ph)
    assert np.array_equal(d_out.cpu().numpy().view(np.uint32), od.view(np.uint32))


def _resampled_guide(guide, pw, ph):
    """ImageShift(guide, 0.5, 0.5) at the positions of NearestResize (DenseUpsampleLayer.cs:98-131), which are sums of 32-bit
    integers: past 32767 rows or columns they wrap below 0, where the reference reads in front of its image and this library
    takes the first row or column."""
    gh, gw, _ = guide.shape

    def taps(n, size):
        acc = (np.arange(n, dtype=np.int64) * int(size * 65536.0 / n)).astype(np.uint32).astype(np.int32)
        return np.clip((acc >> 16)[:, None] - 1 + np.arange(4), 0, size - 1), acc
    rows, ay = taps(ph, gh)
    cols, ax = taps(pw, gw)
    assert ay.min() < 0 or ax.min() < 0
    k = np.array([-1, 9, 9, -1], np.int64)  # sixteenths of the half-pixel cubic taps, exact in the reference's floats
    v = np.einsum("i,yxic->yxc", k, guide.astype(np.int64)[rows.T].transpose(1, 2, 0, 3))
    v = np.einsum("j,yxjc->yxc", k, v[:, cols])
    return np.clip(np.rint(v / 256.0), 0, 255).astype(np.uint8)


@pytest.mark.gpu
@pytest.mark.parametrize("pw,ph", [(16500, 3), (3, 16500), (40000, 2)])
def test_guide_positions_wrap(oracle, pw, ph):
    from lux_b200 import api
    rng = np.random.default_rng(pw + ph)
    depth = rng.uniform(300.0, 6000.0, (ph, pw)).astype(np.float32)
    guide = rng.integers(0, 256, (2 * ph, 2 * pw, 4), dtype=np.uint8)
    g2 = np.ascontiguousarray(_resampled_guide(guide, pw, ph))
    inv, up, want = np.empty_like(depth), np.empty((2 * ph, 2 * pw), np.float32), np.empty((2 * ph, 2 * pw), np.float32)
    L, ptr, i32 = oracle.lib(), (lambda a: ctypes.c_void_p(a.ctypes.data)), ctypes.c_int
    L.lo_inverse_depth(ptr(depth), ctypes.c_size_t(depth.size), ptr(inv))
    L.lo_bilateral_upsample(ptr(inv), i32(pw), i32(ph), ptr(guide), i32(2 * pw), i32(2 * ph), i32(2 * pw), ptr(g2), ctypes.c_float(10.0), ptr(up))
    L.lo_inverse_depth(ptr(up), ctypes.c_size_t(up.size), ptr(want))
    r = api.DenseUpsampleLayer.run(depth, pw, ph, guide, pw, ph, sigma=10.0)
    assert np.array_equal(r.Depth.reshape(want.shape).view(np.uint32), want.view(np.uint32))


# images past the size rule of the quads (the smaller ones above go pixel by pixel): sides of no round size, one of few rows or columns
@pytest.mark.gpu
@pytest.mark.parametrize("pw,ph,with_conf,sigma", [(389, 391, True, 10.0), (389, 391, False, 0.5), (16000, 11, True, 1e-3), (11, 16000, False, 300.0),
                                                   (521, 390, True, 1e10), (521, 390, True, 1e-25)])
def test_many_quads(oracle, pw, ph, with_conf, sigma):
    from lux_b200 import api
    rng = np.random.default_rng(pw + ph)
    depth = rng.uniform(300.0, 6000.0, (ph, pw)).astype(np.float32)
    special = np.array([0.0, -0.0, np.inf, -np.inf, 1e-40, 3e38, -5.0], np.float32)
    depth.reshape(-1)[::7] = np.resize(special, depth.reshape(-1)[::7].size)
    guide = rng.integers(0, 256, (2 * ph, 2 * pw, 4), dtype=np.uint8)
    guide[: ph // 2] = 255
    guide[ph // 2: ph] = rng.integers(0, 2, guide[ph // 2: ph].shape) * 255
    conf = rng.uniform(0, 1, (ph, pw)).astype(np.float32) if with_conf else None
    n0 = api.kernel_launches()
    r = api.DenseUpsampleLayer.run(depth, pw, ph, guide, pw, ph, sigma=sigma, prev_confidence=conf)
    assert api.kernel_launches() - n0 == 3  # resampling, quads and border (an infinite k: depth and confidence pixel by pixel)
    od, oc = oracle.upsample(depth, pw, ph, guide, pw, ph, sigma=sigma, prev_conf=conf)
    got = r.Depth.reshape(od.shape)
    assert ((got.view(np.uint32) == od.view(np.uint32)) | (np.isnan(od) & np.isnan(got))).all()
    if with_conf:
        gc = r.Confidence.reshape(oc.shape)
        assert ((gc.view(np.uint32) == oc.view(np.uint32)) | (np.isnan(oc) & np.isnan(gc))).all()
