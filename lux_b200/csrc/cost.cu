// Plane-sweep matching cost -> u8 raw volume: DenseStereo.MatchingCost + Normalise (DenseStereo.cs:217-292, 376-381).
//
// One warp per reference pixel, lanes over planes. Per other camera and plane: the projection through the flow matrix
// (no FMA, IEEE 1/pz; the plane-only terms z·W2 + W3 come from a per-layer table), the half-pixel `pavgb` resampling
// of the target block, capped |diff| of the 3x3 blocks, the fixed-point channel weights, and a u16 wrap-sum over
// cameras. A plane whose position repeats or leaves the valid rect reuses the last computed cost (:273-274): the warp
// finds that plane with a ballot and carries it across chunks of 32 planes.
//
// Half-pixel phases: the resampled block value at (x, y) with fractions (hx, hy) is pavgb over rows first, then over
// columns, of the 2x2 neighbourhood at (x, y) (:248-253); it depends on (x, y, hx, hy) only, so k_phase_* writes the four
// phase images of every other camera once per layer and a plane's 3x3 block is three row loads with no averaging:
//   grey camera (weights {12240, 0, 0, 0}, only Y contributes): per pixel and phase the Y bytes of columns x, x+1, x+2 in
//     a word, so a block row is one 4-byte load and its differences one instruction, capped at 2 in u16x2 lanes;
//   colour camera: the RGBA word per pixel and phase; even bytes (Y, V) and odd bytes (U, A) as u16x2 lanes.
// Both are exact restatements of the reference's byte-lane sums (each channel sum is at most 9·6).
#include <algorithm>
#include <climits>

#include "common.cuh"
#include "internal.h"

namespace lux {

LUX_DEV uint32_t vmin2c(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("min.u16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
LUX_DEV uint32_t vmax2c(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("max.u16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
LUX_DEV int avg_u8(int a, int b) { return (a + b + 1) >> 1; }                 // pavgb on one byte

// The phase-h value (h = 2·hy + hx) of byte channel `ch` at (x, y): rows averaged first, then columns. Only positions
// whose 2x2 neighbourhood lies in the image are ever read by the cost; the others are clamped.
LUX_DEV int phase_byte(const uint8_t* img, int iw, int ih, int x, int y, int h, int ch) {
  const int x1 = min(x + 1, iw - 1), y1 = min(y + 1, ih - 1);
  auto at = [&](int xx, int yy) { return (int)img[((size_t)yy * iw + xx) * 4 + ch]; };
  int a = at(x, y), b = at(x1, y);
  if (h & 2) {
    a = avg_u8(a, at(x, y1));
    b = avg_u8(b, at(x1, y1));
  }
  return (h & 1) ? avg_u8(a, b) : a;
}

// The two layouts without shared columns: half-pixel position (u, v) = (2x + hx, 2y + hy) at word v·2iw + u, so that a plane's
// block starts one multiply-add away and planes half a pixel apart share their lines; a block's rows are 4iw words apart.
// Grey: the Y bytes of phase 2·hy + hx at columns x, x+1, x+2, low byte first.
__global__ void k_phase_grey(const uint8_t* __restrict__ img, int iw, int ih, uint32_t* __restrict__ out) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y;
  if (x >= iw) return;
  uint32_t v[4];
#pragma unroll
  for (int h = 0; h < 4; h++) {
    const uint32_t p0 = phase_byte(img, iw, ih, x, y, h, 0), p1 = phase_byte(img, iw, ih, min(x + 1, iw - 1), y, h, 0),
                   p2 = phase_byte(img, iw, ih, min(x + 2, iw - 1), y, h, 0);
    v[h] = p0 | p1 << 8 | p2 << 16;
  }
  uint2* o = reinterpret_cast<uint2*>(out) + (size_t)y * 2 * iw + x;
  o[0] = make_uint2(v[0], v[1]);
  o[iw] = make_uint2(v[2], v[3]);
}
// Grey, vertical triples (the shared-column axis kernel): out[h][y][x] = the Y bytes of phase h at rows y, y+1, y+2 of
// column x as u16 pairs: {y | y+2 << 16, y+1}.
__global__ void k_phase_grey_v(const uint8_t* __restrict__ img, int iw, int ih, uint2* __restrict__ out) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y;
  if (x >= iw) return;
#pragma unroll
  for (int h = 0; h < 4; h++) {
    const uint32_t p0 = phase_byte(img, iw, ih, x, y, h, 0), p1 = phase_byte(img, iw, ih, x, min(y + 1, ih - 1), h, 0),
                   p2 = phase_byte(img, iw, ih, x, min(y + 2, ih - 1), h, 0);
    out[((size_t)h * ih + y) * iw + x] = make_uint2(p0 | (p2 << 16), p1);
  }
}
// Colour: the RGBA word of the phase.
__global__ void k_phase_colour(const uint8_t* __restrict__ img, int iw, int ih, uint32_t* __restrict__ out) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y;
  if (x >= iw) return;
  uint32_t v[4];
#pragma unroll
  for (int h = 0; h < 4; h++) {
    v[h] = 0;
#pragma unroll
    for (int ch = 0; ch < 4; ch++) v[h] |= (uint32_t)phase_byte(img, iw, ih, x, y, h, ch) << (8 * ch);
  }
  uint2* o = reinterpret_cast<uint2*>(out) + (size_t)y * 2 * iw + x;
  o[0] = make_uint2(v[0], v[1]);
  o[iw] = make_uint2(v[2], v[3]);
}

// Grey block: S0 = Σ min(|t - r|, 2) over the 3x3 Y block, a row's three bytes in a word (the top bytes are equal: zero).
struct GreyRef {
  uint32_t r[3];
};
LUX_DEV GreyRef grey_ref(const uint32_t (&rb)[3][3]) {
  GreyRef g;
#pragma unroll
  for (int r = 0; r < 3; r++) g.r[r] = (rb[r][0] & 0xffu) | (rb[r][1] & 0xffu) << 8 | (rb[r][2] & 0xffu) << 16;
  return g;
}
LUX_DEV int grey_sum(const uint32_t (&t)[3], const GreyRef& g) {
  const uint32_t v0 = __vabsdiffu4(t[0], g.r[0]), v1 = __vabsdiffu4(t[1], g.r[1]), v2 = __vabsdiffu4(t[2], g.r[2]);
  const uint32_t two = 0x00020002u, m = 0x00ff00ffu;
  const uint32_t s = vmin2c(v0 & m, two) + vmin2c(v1 & m, two) + vmin2c(v2 & m, two) + vmin2c(__byte_perm(v0, v1, 0x3531), two) +
                     vmin2c(__byte_perm(v2, 0, 0x4441), two);  // (byte 3 of a difference is zero)
  return (int)((s & 0xffffu) + (s >> 16));
}
LUX_DEV int grey_weighted(int s0) { return (s0 * 12240 + 16) >> 5; }
LUX_DEV int grey_cost(const uint32_t* __restrict__ q, int iw, const GreyRef& g) {
  const uint32_t t[3] = {__ldg(q), __ldg(q + 4 * (size_t)iw), __ldg(q + 8 * (size_t)iw)};
  return grey_weighted(grey_sum(t, g));
}

// The reference 3x3 block, rows and columns clamped to the image.
LUX_DEV void ref_block(const CostArgs& a, int xImg, int yImg, uint32_t (&rb)[3][3]) {
#pragma unroll
  for (int r = 0; r < 3; r++) {
    const int yy = min(max(yImg + r - 1, 0), a.rh - 1);
#pragma unroll
    for (int c = 0; c < 3; c++)
      rb[r][c] = __ldg(reinterpret_cast<const uint32_t*>(a.ref) + (size_t)yy * a.rw + min(max(xImg + c - 1, 0), a.rw - 1));
  }
}

// Colour block: the four bytes' differences at once, then {Y, V} of a pixel and {U, U} of two as u16 pairs, capped at {2, 6}
// and 6. A's cap is 0, so its sum is, and (0·w + 16) >> 5 adds nothing.
LUX_DEV int colour_cost(const uint32_t* __restrict__ q, int iw, const uint32_t (&rb)[3][3], const uint16_t (&wq)[4]) {
  uint32_t v[9], se = 0, so = 0;
#pragma unroll
  for (int i = 0; i < 9; i++) v[i] = __ldg(q + (size_t)(i / 3) * 4 * iw + 2 * (i % 3));
#pragma unroll
  for (int i = 0; i < 9; i++) {
    v[i] = __vabsdiffu4(v[i], rb[i / 3][i % 3]);
    se += vmin2c(v[i] & 0x00ff00ffu, 0x00060002u);
  }
#pragma unroll
  for (int i = 0; i < 8; i += 2) so += vmin2c(__byte_perm(v[i], v[i + 1], 0x5511) & 0x00ff00ffu, 0x00060006u);
  so += min((v[8] >> 8) & 0xffu, 6u);
  const int S0 = se & 0xffff, S2 = se >> 16, S1 = (so & 0xffff) + (so >> 16);
  const int cY = (S0 * wq[0] + 16) >> 5, cU = (S1 * wq[1] + 16) >> 5, cV = (S2 * wq[2] + 16) >> 5;
  return cY + cU + cV;  // at most 6885: MathF.Min(…, 65535) and the float round trip change nothing
}

template <bool GREY>
__global__ void __launch_bounds__(256) k_cost(const CostArgs a, const LayerGeom g, const float4* __restrict__ zt,
                                              uint8_t* __restrict__ raw, int* err) {
  __shared__ int s_carry[8][kMaxCams];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  const int npx = g.W * g.H;
  const int n = g.n_planes;
  const int half = (a.scale + (a.scale >> 31)) >> 1;
  for (int pi = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; pi < npx; pi += nwarps) {
    if (g.skip[pi]) {  // skipped pixels aggregate raw 0 and 255 past their count (DenseStereoSgm.cs:242)
      uint8_t* out = raw + g.off[pi];
      const int count = g.count[pi], cap = g.cap[pi];
      for (int d = lane; d < cap; d += 32) out[d] = d < count ? 0 : 255;
      continue;
    }
    const int x = pi % g.W, y = pi / g.W;
    const int xImg = min(a.scale * x + half, a.rw - 1), yImg = min(a.scale * y + half, a.rh - 1);
    const int start = g.start[pi], count = g.count[pi], cap = g.cap[pi];
    uint8_t* out = raw + g.off[pi];
    if (start + count > n) {  // MatchingCostScalar would index Planes past its end
      if (lane == 0) atomicCAS(err, 0, 7);
      continue;
    }
    uint32_t rb[3][3];
    ref_block(a, xImg, yImg, rb);
    const GreyRef gr = grey_ref(rb);
    const float xf = (float)xImg, yf = (float)yImg;
    for (int c0 = 0; c0 < count; c0 += 32) {
      const int d = c0 + lane;
      const bool valid = d < count;
      const int pl = valid ? start + d : start;
      const float z = __ldg(g.planes + pl);
      const int last = min(31, count - 1 - c0);
      const float xz = __fmul_rn(xf, z), yz = __fmul_rn(yf, z);  // (x·z)·1.0f: the product by one is exact
      uint32_t acc = 0;
      for (int k = 0; k < a.n_others; k++) {
        const float* Wm = a.warp[k];
        const int iw = a.ow[k], ih = a.oh[k];
        const int x0 = 1, y0 = 1, x1 = iw - 2, y1 = ih - 2;
        // p = ((z·W2 + W3) + xz·W0) + yz·W1 (:255-259), the first term from the table; then 1/pz and the +0.25 bias
        const float4 zk = __ldg(zt + (size_t)k * n + pl);
        const float px = __fadd_rn(__fadd_rn(zk.x, __fmul_rn(xz, Wm[0])), __fmul_rn(yz, Wm[4]));
        const float py = __fadd_rn(__fadd_rn(zk.y, __fmul_rn(xz, Wm[1])), __fmul_rn(yz, Wm[5]));
        const float pz = __fadd_rn(__fadd_rn(zk.z, __fmul_rn(xz, Wm[2])), __fmul_rn(yz, Wm[6]));
        const float inv = __frcp_rn(pz);  // the correctly rounded 1/pz, as the reference's division
        float fx = __fadd_rn(__fmul_rn(px, inv), 0.25f), fy = __fadd_rn(__fmul_rn(py, inv), 0.25f);
        if (d == 0) {  // the first plane is clamped into the rect (:263-269)
          fx = cs_minf(cs_maxf(fx, (float)x0), (float)(x1 - 1));
          fy = cs_minf(cs_maxf(fy, (float)y0), (float)(y1 - 1));
        }
        // (int)(2f) gives the integer part (>> 1) and the half-pixel bit (& 1) wherever the position can be in the rect
        // (f >= 1); elsewhere both forms fall outside it
        const int tx = f2i(__fadd_rn(fx, fx)), ty = f2i(__fadd_rn(fy, fy));
        const int ix = tx >> 1, iy = ty >> 1;
        bool inb = valid && !(ix < x0 || ix >= x1 || iy < y0 || iy >= y1);
        if (d == 0 && !inb) {  // the scalar fallback of the reference would read out of the image
          atomicCAS(err, 0, 7);
        }
        int costK = 0;
        if (inb) {
          const size_t qi = (size_t)(ty - 2) * (2 * iw) + (tx - 2);
          if (GREY) costK = grey_cost(a.phase[k] + qi, iw, gr);
          else costK = colour_cost(a.phase[k] + qi, iw, rb, a.wq[k]);
        }
        const uint32_t m = __ballot_sync(0xffffffffu, inb);
        const uint32_t below = m & ((1u << lane) - 1u);
        const int src = below ? 31 - __clz(below) : 0;
        const int prevCost = __shfl_sync(0xffffffffu, costK, src);
        const int carry = c0 == 0 ? 0 : s_carry[wib][k];
        const int res = inb ? costK : (below ? prevCost : carry);
        __syncwarp();
        const int tail = __shfl_sync(0xffffffffu, res, last);
        if (lane == 0) s_carry[wib][k] = tail;
        __syncwarp();
        acc += (uint32_t)res;
      }
      if (valid) out[d] = (uint8_t)f2i(__fmul_rn((float)(acc & 0xffffu), a.norm));  // Normalise (:378-379)
    }
    for (int d = count + lane; d < cap; d += 32) out[d] = 255;  // padding planes (:380)
  }
}

// Uniform layers (every pixel searches planes [0, n), cap n, n % 8 == 0; 1 to 15 other cameras): lanes over 32
// neighbouring pixels of a row, each walking its pixel's planes in order like the reference's loop. Eight planes at a time
// go through camera after camera: the camera's constants, its last computed cost (:273-274, kept in shared memory between
// the eights) and the lines of its phase images are then in hand for eight planes, and eight costs go out in one store. Four
// positions are projected and their blocks loaded together, unless no lane of the warp hits the camera's rect with any of
// them. Bound by issue (57 instructions a camera and plane): ten grey cameras of 2080x1560 D=176 11.2 ms; with the cameras
// inside the plane loop, and u16 pairs of twice the bytes, it took 22.7 (95 instructions, an eighth of the sectors from L1).
// Skipped pixels get raw 0 (DenseStereoSgm.cs:242).
constexpr int kRowsThreads = 128;
template <bool GREY>
__global__ void __launch_bounds__(kRowsThreads) k_cost_rows(const __grid_constant__ CostArgs a, const LayerGeom g, const float4* __restrict__ zt,
                                                   uint8_t* __restrict__ raw, int* err) {
  __shared__ uint16_t s_last[kMaxCams][kRowsThreads];
  const int lane = threadIdx.x & 31;
  const int tiles_x = (g.W + 31) >> 5;
  const int ntiles = tiles_x * g.H;
  const int n = g.n_planes;
  const int half = (a.scale + (a.scale >> 31)) >> 1;
  const int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (t < ntiles) {
    const int y = t / tiles_x, xr = ((t - y * tiles_x) << 5) + lane, x = min(xr, g.W - 1);
    const size_t pi = (size_t)y * g.W + x;
    uint8_t* out = raw + pi * n;
    const bool skipped = g.skip[pi] != 0, live = xr < g.W && !skipped;
    if (xr < g.W && skipped)
      for (int d = 0; d < n; d += 8) *reinterpret_cast<uint2*>(out + d) = make_uint2(0u, 0u);
    if (!__any_sync(0xffffffffu, live)) return;
    const int xImg = min(a.scale * x + half, a.rw - 1), yImg = min(a.scale * y + half, a.rh - 1);
    uint32_t rb[3][3];
    ref_block(a, xImg, yImg, rb);
    const GreyRef gr = grey_ref(rb);
    const float xf = (float)xImg, yf = (float)yImg;
    for (int d0 = 0; d0 < n; d0 += 8) {
      float xz[8], yz[8];
      uint32_t acc[8];
#pragma unroll
      for (int j = 0; j < 8; j++) {
        const float z = __ldg(g.planes + d0 + j);
        xz[j] = __fmul_rn(xf, z);
        yz[j] = __fmul_rn(yf, z);
        acc[j] = 0;
      }
#pragma unroll 1
      for (int k = 0; k < a.n_others; k++) {
        const float* Wm = a.warp[k];
        const float w0 = Wm[0], w1 = Wm[1], w2 = Wm[2], w4 = Wm[4], w5 = Wm[5], w6 = Wm[6];
        const int iw = a.ow[k], ih = a.oh[k];
        const unsigned wide = (unsigned)max(2 * iw - 6, 0), high = (unsigned)max(2 * ih - 6, 0), pitch = 2 * (unsigned)iw;  // in half pixels
        const uint32_t* phase = a.phase[k];
        const float4* zk = zt + (size_t)k * n + d0;
        int last = d0 > 0 ? s_last[k][threadIdx.x] : 0;
#pragma unroll
        for (int q = 0; q < 8; q += 4) {
          float px[4], py[4], pz[4];
#pragma unroll
          for (int j = 0; j < 4; j++) {
            const float4 zj = __ldg(zk + q + j);
            px[j] = __fadd_rn(__fadd_rn(zj.x, __fmul_rn(xz[q + j], w0)), __fmul_rn(yz[q + j], w4));
            py[j] = __fadd_rn(__fadd_rn(zj.y, __fmul_rn(xz[q + j], w1)), __fmul_rn(yz[q + j], w5));
            pz[j] = __fadd_rn(__fadd_rn(zj.z, __fmul_rn(xz[q + j], w2)), __fmul_rn(yz[q + j], w6));
          }
          float inv[4];
          const float big = fmaxf(fmaxf(fabsf(pz[0]), fabsf(pz[1])), fmaxf(fabsf(pz[2]), fabsf(pz[3])));
          const float small = fminf(fminf(fabsf(pz[0]), fabsf(pz[1])), fminf(fabsf(pz[2]), fabsf(pz[3])));
          if (big < 0x1p125f && small >= 0x1p-125f) {
#pragma unroll
            for (int j = 0; j < 4; j++) inv[j] = rcp_mid(pz[j]);
          } else {
#pragma unroll
            for (int j = 0; j < 4; j++) inv[j] = __frcp_rn(pz[j]);
          }
          int at[4];  // where the block starts in the phase images, -1 outside the rect
#pragma unroll
          for (int j = 0; j < 4; j++) {
            float fx = __fadd_rn(__fmul_rn(px[j], inv[j]), 0.25f), fy = __fadd_rn(__fmul_rn(py[j], inv[j]), 0.25f);
            if (q + j == 0 && d0 == 0) {  // the first plane is clamped into the rect (:263-269)
              fx = cs_minf(cs_maxf(fx, 1.0f), (float)(iw - 3));
              fy = cs_minf(cs_maxf(fy, 1.0f), (float)(ih - 3));
            }
            // (int)(2f) - 2, the half-pixel position of the block's first row and column: the low bits of 2f + 1.5·2^23 rounded
            // toward zero wherever the position can be in the rect, and past every rect for all other floats and NaN
            const unsigned u = __float_as_uint(__fmaf_rz(fx, 2.0f, 12582912.0f)) - 0x4b400002u, v = __float_as_uint(__fmaf_rz(fy, 2.0f, 12582912.0f)) - 0x4b400002u;
            const bool in = u < wide && v < high;
            at[j] = in ? (int)(v * pitch + u) : -1;
            // the scalar fallback of the reference would read out of the image
            if (q + j == 0 && d0 == 0 && !in && live) atomicCAS(err, 0, 7);
          }
          if (!__any_sync(0xffffffffu, (at[0] & at[1] & at[2] & at[3]) >= 0)) {
#pragma unroll
            for (int j = 0; j < 4; j++) acc[q + j] += (uint32_t)last;
            continue;
          }
          if (GREY) {
            uint32_t w[4][3];
#pragma unroll
            for (int j = 0; j < 4; j++) {
              const uint32_t* b = phase + max(at[j], 0);
#pragma unroll
              for (int r = 0; r < 3; r++) w[j][r] = __ldg(b + r * 2 * pitch);
            }
#pragma unroll
            for (int j = 0; j < 4; j++) {
              const int c = grey_weighted(grey_sum(w[j], gr));
              last = at[j] >= 0 ? c : last;
              acc[q + j] += (uint32_t)last;
            }
          } else {
#pragma unroll
            for (int j = 0; j < 4; j++) {
              if (at[j] >= 0) last = colour_cost(phase + at[j], iw, rb, a.wq[k]);
              acc[q + j] += (uint32_t)last;
            }
          }
        }
        s_last[k][threadIdx.x] = (uint16_t)last;
      }
      uint32_t pk[2] = {0, 0};
#pragma unroll
      for (int j = 0; j < 8; j++)  // Normalise (:378-379)
        pk[j >> 2] |= ((uint32_t)f2i(__fmul_rn((float)(acc[j] & 0xffffu), a.norm)) & 0xffu) << (8 * (j & 3));
      if (live) *reinterpret_cast<uint2*>(out + d0) = make_uint2(pk[0], pk[1]);
    }
  }
}

// Uniform layers of one axis-aligned camera pair (flow-matrix terms W1 = W2 = W4 = W6 = 0, as for a rectified pair; the
// host checks them, that every plane term z·W10 + W14 is finite and non-zero and that x·z cannot overflow). Then, exactly:
//   pz = z·W10 + W14 (adding the ±0 products changes no non-zero value), so 1/pz is a per-plane constant (zt.w);
//   px = (z·W8 + W12) + x·z·W0, where the dropped ±0 term can only change the sign of a zero px, and a zero px gives
//     the same fx (0.25, or NaN with an infinite 1/pz) either way;
//   py = (z·W9 + W13) + y·z·W5 likewise, so the row and half-pixel bit of the target depend on (row, plane) only: lane j
//     of a warp computes them for plane d0 + j and the warp shuffles them to every pixel.
// The first plane (clamped into the rect) keeps the general projection.
template <bool GREY>
__global__ void __launch_bounds__(256) k_cost_axis(const CostArgs a, const LayerGeom g, const float4* __restrict__ zt,
                                                   uint8_t* __restrict__ raw, int* err) {
  const int lane = threadIdx.x & 31;
  const int tiles_x = (g.W + 31) >> 5;
  const int ntiles = tiles_x * g.H;
  const int n = g.n_planes;
  const int half = (a.scale + (a.scale >> 31)) >> 1;
  const float* Wm = a.warp[0];
  const float w0 = Wm[0], w1 = Wm[1], w2 = Wm[2], w4 = Wm[4], w5 = Wm[5], w6 = Wm[6];
  const int iw = a.ow[0], ih = a.oh[0], x1 = iw - 2, y1 = ih - 2;
  const uint32_t* phase = a.phase[0];
  constexpr int kNoRow = INT_MIN;
  for (int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < ntiles; t += (gridDim.x * blockDim.x) >> 5) {
    const int y = t / tiles_x, xr = ((t - y * tiles_x) << 5) + lane;
    const int x = min(xr, g.W - 1);
    const size_t pi = (size_t)y * g.W + x;
    uint8_t* out = raw + pi * n;
    const bool skipped = g.skip[pi] != 0;
    const bool live = xr < g.W && !skipped;
    if (xr < g.W && skipped)
      for (int d = 0; d < n; d += 8) *reinterpret_cast<uint2*>(out + d) = make_uint2(0u, 0u);
    if (__ballot_sync(0xffffffffu, live) == 0) continue;
    const int xImg = min(a.scale * x + half, a.rw - 1), yImg = min(a.scale * y + half, a.rh - 1);
    uint32_t rb[3][3];
    ref_block(a, xImg, yImg, rb);
    const GreyRef gr = grey_ref(rb);
    const float xf = (float)xImg, yf = (float)yImg;
    int last = 0;
    uint32_t pk0 = 0, pk1 = 0;
    auto put = [&](int d, uint32_t acc) {  // Normalise (:378-379) and eight planes per store
      const uint32_t b = (uint32_t)f2i(__fmul_rn((float)(acc & 0xffffu), a.norm)) & 0xffu;
      const int sh = (d & 3) * 8;
      if (d & 4) pk1 |= b << sh;
      else pk0 |= b << sh;
      if ((d & 7) == 7) {
        if (live) *reinterpret_cast<uint2*>(out + (d - 7)) = make_uint2(pk0, pk1);
        pk0 = pk1 = 0;
      }
    };
    {  // plane 0: the general projection, clamped into the rect (:263-269)
      const float z = __ldg(g.planes);
      const float xz = __fmul_rn(xf, z), yz = __fmul_rn(yf, z);
      const float4 zk = __ldg(zt);
      const float px = __fadd_rn(__fadd_rn(zk.x, __fmul_rn(xz, w0)), __fmul_rn(yz, w4));
      const float py = __fadd_rn(__fadd_rn(zk.y, __fmul_rn(xz, w1)), __fmul_rn(yz, w5));
      const float pz = __fadd_rn(__fadd_rn(zk.z, __fmul_rn(xz, w2)), __fmul_rn(yz, w6));
      const float inv = __frcp_rn(pz);
      const float fx = cs_minf(cs_maxf(__fadd_rn(__fmul_rn(px, inv), 0.25f), 1.0f), (float)(x1 - 1));
      const float fy = cs_minf(cs_maxf(__fadd_rn(__fmul_rn(py, inv), 0.25f), 1.0f), (float)(y1 - 1));
      const int tx = f2i(__fadd_rn(fx, fx)), ty = f2i(__fadd_rn(fy, fy));
      const int ix = tx >> 1, iy = ty >> 1;
      if (ix >= 1 && ix < x1 && iy >= 1 && iy < y1) {
        if (live) {
          const size_t qi = (size_t)(ty - 2) * (2 * iw) + (tx - 2);
          last = GREY ? grey_cost(phase + qi, iw, gr) : colour_cost(phase + qi, iw, rb, a.wq[0]);
        }
      } else if (live) {  // the scalar fallback of the reference would read out of the image
        atomicCAS(err, 0, 7);
      }
      put(0, (uint32_t)last);
    }
    for (int d0 = 0; d0 < n; d0 += 32) {
      // lane j: the target row offset of plane d0 + j (or kNoRow when the row leaves the rect)
      int rowoff;
      {
        const int dj = min(d0 + lane, n - 1);
        const float4 zj = __ldg(zt + dj);
        const float yz = __fmul_rn(yf, __ldg(g.planes + dj));
        const float fy = __fadd_rn(__fmul_rn(__fadd_rn(zj.y, __fmul_rn(yz, w5)), zj.w), 0.25f);
        const int ty = f2i(__fadd_rn(fy, fy)), iy = ty >> 1;
        rowoff = (iy >= 1 && iy < y1) ? (ty - 2) * 2 * iw - 2 : kNoRow;
      }
      const int jend = min(32, n - d0);
      for (int j = (d0 == 0 ? 1 : 0); j < jend; j++) {
        const int d = d0 + j;
        const int ro_d = __shfl_sync(0xffffffffu, rowoff, j);
        if (ro_d != kNoRow && live) {
          const float4 zk = __ldg(zt + d);
          const float xz = __fmul_rn(xf, __ldg(g.planes + d));
          const float fx = __fadd_rn(__fmul_rn(__fadd_rn(zk.x, __fmul_rn(xz, w0)), zk.w), 0.25f);
          const int tx = f2i(__fadd_rn(fx, fx)), ix = tx >> 1;
          if (ix >= 1 && ix < x1) {
            const int qi = ro_d + tx;
            last = GREY ? grey_cost(phase + qi, iw, gr) : colour_cost(phase + qi, iw, rb, a.wq[0]);
          }
        }
        put(d, (uint32_t)last);
      }
    }
  }
}

// One block column of the grey cost: the three capped differences of a target column triple t (vertical layout) against
// a reference column triple, in u16x2 lanes each offset by 256 (as grey_cost); three columns sum to S0 + 12·256.
struct ColRef {
  uint32_t ea, eb, oa, ob;
};
LUX_DEV ColRef col_ref(uint32_t even, uint32_t odd) { return ColRef{0x01000100u - even, 0x01000100u + even, 0x01000100u - odd, 0x01000100u + odd}; }
LUX_DEV uint32_t col_cost(uint2 t, const ColRef& c) {
  return vmin2c(vmax2c(t.x + c.ea, c.eb - t.x), 0x01020102u) + vmin2c(vmax2c(t.y + c.oa, c.ob - t.y), 0x01000102u);
}
// The same with the four adds as multiply-adds by one = 1 and neg = 0xffffffff (kernel-argument values, so they stay
// multiply-adds and issue on the FMA pipe; the ALU pipe bounds the kernel that uses this). Equal mod 2^32.
LUX_DEV uint32_t col_cost_m(uint2 t, const ColRef& c, uint32_t one, uint32_t neg) {
  return vmin2c(vmax2c(t.x * one + c.ea, t.x * neg + c.eb), 0x01020102u) +
         vmin2c(vmax2c(t.y * one + c.oa, t.y * neg + c.ob), 0x01000102u);
}

// Uniform layers of one axis-aligned grey pair at scale 1 (the plain stereo pair): the 3x3 blocks of neighbouring
// pixels overlap, and so do their target blocks wherever the target column advances by one whole pixel with the same
// half-pixel phase from one pixel to the next. A lane holds P neighbouring pixels of a row (slots 0..P-1) and a warp a
// run of 32·P - 2 pixels (slots 0 and 1 of lane 0 are the two pixels to the left of the run, computed and not stored).
// Per plane every slot computes only the right column of its block (reference column x + 1, clamped as the reference
// clamps its block, against target column ix + 1) and takes the middle and left columns from the two pixels to its left
// (the lane's own slots, or slots P-2 and P-1 of the lane to the left by shuffle) when their target positions are
// exactly 2 and 4 half-pixels to the left; a warp vote keeps the common case, where every slot that needs its block has
// it that way, free of per-slot branches. Elsewhere a slot computes the two columns itself. The terms, and so the sums,
// are the reference's (:222-246); only who computes a term changes. The plane terms, the target row and the neighbour
// exchange are shared by the lane's P pixels. Normalise (:378-379) of one camera's cost is a function of S0 (0..18), a
// 19-entry table. Two pixels a lane: 4 (79 registers) take more issue slots a DE, and staging each 32-plane group in
// shared memory (whole-sector stores) saves DRAM traffic the kernel is not bound by at the price of instructions it is.
constexpr int kAxPx = 2;                 // pixels a lane
constexpr int kAxRun = 32 * kAxPx - 2;  // pixels a warp stores

template <int P>
__global__ void __launch_bounds__(256, P > 2 ? 3 : 4)
    k_cost_axis_v(const CostArgs a, const LayerGeom g, const float4* __restrict__ zt, uint8_t* __restrict__ raw, int* err) {
  constexpr int kRun = 32 * P - 2;
  __shared__ uint8_t s_norm[32];
  if (threadIdx.x < 32)
    s_norm[threadIdx.x] =
        (uint8_t)(f2i(__fmul_rn((float)(((uint32_t)(min((int)threadIdx.x, 18) * 12240 + 16) >> 5) & 0xffffu), a.norm)) & 0xff);
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int runs_x = (g.W + kRun - 1) / kRun;
  const int nruns = runs_x * g.H;
  const int n = g.n_planes;
  const uint8_t* ref8 = a.ref;
  const float* Wm = a.warp[0];
  const float w0 = Wm[0], w1 = Wm[1], w2 = Wm[2], w4 = Wm[4], w5 = Wm[5], w6 = Wm[6];
  const int iw = a.ow[0], ih = a.oh[0], x1 = iw - 2, y1 = ih - 2;
  const uint2* q = reinterpret_cast<const uint2*>(a.phase[0]);
  const int plane_stride = ih * iw;
  constexpr int kNoRow = INT_MIN;
  // (s · 0x10001) >> 16 is the sum of the two u16 lanes of a block sum s (each lane under 2^15, so nothing carries)
  const uint32_t one = a.one, neg = 0u - a.one, k10001 = 0x10001u * a.one;
  for (int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < nruns; t += (gridDim.x * blockDim.x) >> 5) {
    const int y = t / runs_x;
    const int x0 = (t - y * runs_x) * kRun - 2;  // x of slot 0 of lane 0
    const int xs = x0 + lane * P;                // x of this lane's slot 0
    const long long row0 = (long long)y * g.W;
    bool live[P];
    float xf[P];
    ColRef cr[P];
    const int ya = max(y - 1, 0), yb = min(y + 1, a.rh - 1);
    bool any = false;
#pragma unroll
    for (int j = 0; j < P; j++) {
      const int x = xs + j;
      const bool in_row = lane * P + j >= 2 && x < g.W;  // slots 0 and 1 of lane 0 belong to the run to the left
      const bool skipped = in_row && g.skip[row0 + x] != 0;
      live[j] = in_row && !skipped;
      any = any || live[j];
      if (skipped) {  // skipped pixels aggregate raw 0 (DenseStereoSgm.cs:242)
        uint8_t* out = raw + (row0 + x) * n;
        for (int d = 0; d < n; d += 8) *reinterpret_cast<uint2*>(out + d) = make_uint2(0u, 0u);
      }
      xf[j] = (float)min(x, a.rw - 1);  // scale 1: the reference grid is the layer grid
      // this slot's right reference column (rows y-1, y, y+1 and the column clamped like the reference's block)
      const int c = min(max(x + 1, 0), a.rw - 1);
      const uint32_t r0 = ref8[((size_t)ya * a.rw + c) * 4], r1 = ref8[((size_t)y * a.rw + c) * 4], r2 = ref8[((size_t)yb * a.rw + c) * 4];
      cr[j] = col_ref(r0 | (r2 << 16), r1);
    }
    if (__ballot_sync(0xffffffffu, any) == 0) continue;
    // slots P-2 and P-1 of the lane to the left. Slot j's left and middle block columns are entries j and j + 1 of
    // {left lane's P-2, left lane's P-1, own 0, ..., own P-1}, its right column entry j + 2.
    const ColRef lA{__shfl_up_sync(0xffffffffu, cr[P - 2].ea, 1), __shfl_up_sync(0xffffffffu, cr[P - 2].eb, 1),
                    __shfl_up_sync(0xffffffffu, cr[P - 2].oa, 1), __shfl_up_sync(0xffffffffu, cr[P - 2].ob, 1)};
    const ColRef lB{__shfl_up_sync(0xffffffffu, cr[P - 1].ea, 1), __shfl_up_sync(0xffffffffu, cr[P - 1].eb, 1),
                    __shfl_up_sync(0xffffffffu, cr[P - 1].oa, 1), __shfl_up_sync(0xffffffffu, cr[P - 1].ob, 1)};
    auto ext_ref = [&](int e) -> const ColRef& { return e == 0 ? lA : e == 1 ? lB : cr[e - 2]; };
    uint32_t last[P];  // the normalised cost of the last plane computed, per slot (:273-274)
    {  // plane 0: the general projection, clamped into the rect (:263-269)
      const float z = __ldg(g.planes);
      const float4 zk = __ldg(zt);
      const float yz = __fmul_rn((float)y, z);
#pragma unroll
      for (int j = 0; j < P; j++) {
        last[j] = 0;
        const float xz = __fmul_rn(xf[j], z);
        const float px = __fadd_rn(__fadd_rn(zk.x, __fmul_rn(xz, w0)), __fmul_rn(yz, w4));
        const float py = __fadd_rn(__fadd_rn(zk.y, __fmul_rn(xz, w1)), __fmul_rn(yz, w5));
        const float pz = __fadd_rn(__fadd_rn(zk.z, __fmul_rn(xz, w2)), __fmul_rn(yz, w6));
        const float inv = __frcp_rn(pz);
        const float fx = cs_minf(cs_maxf(__fadd_rn(__fmul_rn(px, inv), 0.25f), 1.0f), (float)(x1 - 1));
        const float fy = cs_minf(cs_maxf(__fadd_rn(__fmul_rn(py, inv), 0.25f), 1.0f), (float)(y1 - 1));
        const int tx = f2i(__fadd_rn(fx, fx)), ty = f2i(__fadd_rn(fy, fy));
        const int ix = tx >> 1, iy = ty >> 1;
        if (ix >= 1 && ix < x1 && iy >= 1 && iy < y1) {
          if (live[j]) {
            const size_t base = ((size_t)(((ty & 1) << 1) | (tx & 1)) * ih + (iy - 1)) * iw + (ix - 1);
            const uint32_t s = col_cost(__ldg(q + base), ext_ref(j)) + col_cost(__ldg(q + base + 1), ext_ref(j + 1)) +
                               col_cost(__ldg(q + base + 2), cr[j]);
            last[j] = s_norm[(s & 0xffffu) + (s >> 16) - 12 * 256];
          }
        } else if (live[j]) {  // the scalar fallback of the reference would read out of the image
          atomicCAS(err, 0, 7);
        }
      }
    }
    const float yf = (float)y;
    auto row_offset = [&](int d) {  // lane j: the offset of row iy - 1 of phase 2·hy of plane d + j (kNoRow: off the rect)
      const int dj = min(d + lane, n - 1);
      const float4 zj = __ldg(zt + dj);
      const float yz = __fmul_rn(yf, __ldg(g.planes + dj));
      const float fy = __fadd_rn(__fmul_rn(__fadd_rn(zj.y, __fmul_rn(yz, w5)), zj.w), 0.25f);
      const int ty = f2i(__fadd_rn(fy, fy)), iy = ty >> 1;
      return (iy >= 1 && iy < y1) ? (((ty & 1) << 1) * ih + iy - 1) * iw : kNoRow;
    };
    int rowoff = row_offset(0);
    // eight planes of u8 costs a slot as one 64-bit value {lo, hi}, plane d at byte d % 8: each plane shifts it right by
    // one byte and enters at the top
    uint32_t lo[P], hi[P];
#pragma unroll
    for (int j = 0; j < P; j++) {
      lo[j] = 0;
      hi[j] = last[j] << 24;
    }
    for (int d = 1; d < n; d++) {
      if ((d & 31) == 0) rowoff = row_offset(d);
      const int ro_d = __shfl_sync(0xffffffffu, rowoff, d & 31);
      if (ro_d != kNoRow) {  // the same for the whole warp
        const float4 zk = __ldg(zt + d);
        const float z = __ldg(g.planes + d);
        int tx[P], ix[P], rb[P];
        uint32_t c[P];
        bool inr[P];
#pragma unroll
        for (int j = 0; j < P; j++) {
          const float xz = __fmul_rn(xf[j], z);
          const float fx = __fadd_rn(__fmul_rn(__fadd_rn(zk.x, __fmul_rn(xz, w0)), zk.w), 0.25f);
          tx[j] = f2i(__fadd_rn(fx, fx));
          ix[j] = tx[j] >> 1;
          inr[j] = ix[j] >= 1 && ix[j] < x1;
          rb[j] = ro_d + (tx[j] & 1) * plane_stride;  // row iy - 1 of the slot's phase
          // column ix + 1, clamped only to stay in the image: a column a neighbour takes (ix + 1 of a slot whose right
          // neighbour is in the rect one pixel on) lies in [0, iw - 3] already, so a negative ix + 1 may map to iw - 1
          c[j] = col_cost_m(__ldg(q + rb[j] + min((uint32_t)(ix[j] + 1), (uint32_t)(iw - 1))), cr[j], one, neg);
        }
        // slots P-2 and P-1 of the lane to the left; slot P-1's target is sent as kNoRow unless slot P-2's is one pixel
        // left of it, so that one comparison checks both neighbours of slot 0. A neighbour pair found unequal (by this
        // or by the wrapping compares below) only sends a slot to its own columns, which is always exact.
        const int tl = (uint32_t)tx[P - 1] - (uint32_t)tx[P - 2] == 2u ? tx[P - 1] : kNoRow;
        const uint32_t cA = __shfl_up_sync(0xffffffffu, c[P - 2], 1), cB = __shfl_up_sync(0xffffffffu, c[P - 1], 1);
        const int tB = __shfl_up_sync(0xffffffffu, tl, 1);
        bool fast[P];
        bool pair[P];  // pair[j]: slot j's target is one pixel right of slot j-1's (j >= 1)
#pragma unroll
        for (int j = 1; j < P; j++) pair[j] = (uint32_t)tx[j] - (uint32_t)tx[j - 1] == 2u;
        fast[0] = (uint32_t)tx[0] - (uint32_t)tB == 2u;
#pragma unroll
        for (int j = 1; j < P; j++) fast[j] = pair[j] && (j == 1 ? fast[0] : pair[j - 1]);
        bool ok = true;  // every slot that needs its block has it from its neighbours
#pragma unroll
        for (int j = 0; j < P; j++) ok = ok && (fast[j] || !(live[j] && inr[j]));
        auto ext_c = [&](int e) { return e == 0 ? cA : e == 1 ? cB : c[e - 2]; };
        if (__all_sync(0xffffffffu, ok)) {
#pragma unroll
          for (int j = 0; j < P; j++) {
            const uint32_t sum = ext_c(j) + ext_c(j + 1) + c[j];
            if (inr[j]) last[j] = s_norm[((sum * k10001) >> 16) - 12 * 256];
          }
        } else {
#pragma unroll
          for (int j = 0; j < P; j++) {
            if (inr[j]) {
              uint32_t sum;
              if (fast[j]) sum = ext_c(j) + ext_c(j + 1) + c[j];
              else sum = col_cost(__ldg(q + rb[j] + ix[j] - 1), ext_ref(j)) + col_cost(__ldg(q + rb[j] + ix[j]), ext_ref(j + 1)) + c[j];
              last[j] = s_norm[(sum & 0xffffu) + (sum >> 16) - 12 * 256];
            }
          }
        }
      }
#pragma unroll
      for (int j = 0; j < P; j++) {
        lo[j] = __funnelshift_r(lo[j], hi[j], 8);
        hi[j] = __funnelshift_r(hi[j], last[j], 8);
      }
      if ((d & 7) == 7) {
        const int d0 = d - 7;
#pragma unroll
        for (int j = 0; j < P; j++)
          if (live[j]) *reinterpret_cast<uint2*>(raw + (row0 + xs + j) * n + d0) = make_uint2(lo[j], hi[j]);
      }
    }
  }
}

// ---------------- an axis-aligned grey pair of one focal length at scale 1 ----------------
//
// Every target then lies a whole number of half pixels from its pixel, the same number along a row and along a column for
// most planes; rounding tips positions of a plane whose shift falls near the middle of two half pixels to one or the other.
// k_unit_planes evaluates the reference's projection for every column and every row of every plane and records, per plane,
// the shift in half pixels and the interval of in-rect columns and rows, or that two shifts occur, or more.
//
// k_cost_unit then works on bytes, four neighbouring pixels a word: |t - r| by the byte-wise absolute difference, capped at
// 2, summed over the three rows, then over three columns (the neighbouring bytes; from the lanes beside at a word's ends):
// at most 18, no carry. The normalised cost is one multiply of two sums a word (cost_unit_norm). A warp (a block by itself,
// so that the plane's scalars and the row addresses stay on the uniform datapath) takes a run of 120
// pixels (lanes 0 and 31 only supply their columns) of kUnitRows rows, sharing the capped differences of the rows between
// them, and 32 planes at a time through shared memory, so that a pixel's costs go out in 32-byte pieces. A plane of two
// shifts makes the costs of both and selects by each pixel's own target; plane 0 (clamped into the rect) and planes of more
// gather each block by itself. The byte phase images come in four copies, each a byte further on, so that every word load
// is aligned. Bound by the ALU pipe (64 operations a plane, row and warp: 128 pixels): 4160x3120 D=256 takes 2.2 ms
// (k_cost_axis_v 7.7), 2080x1560 D=256 0.61 (1.97), 1040x780 D=64 0.080 (0.163). Three rows a warp: 2.1, 0.65, 0.089.
constexpr int kUnitRows = 2, kUnitRun = 120, kUnitPad = 256;
__host__ __device__ constexpr int unit_pitch(int w) { return (w + 2 * kUnitPad + 127) & ~127; }
struct UnitPlane {
  int dx, xa, xb;  // columns xa..xb-1 are in the rect, 2·column + dx half pixels (or dx + 1 where two_x)
  int dy, ya, yb;  // rows likewise
  int two_x, two_y;
  int whole;       // the intervals and shifts say it all
  int other;       // more shifts than two, or gaps in an interval
  int pad[2];
};

int cost_unit_tiles(int W, int H) { return ((W + kUnitRun - 1) / kUnitRun) * ((H + kUnitRows - 1) / kUnitRows); }
size_t cost_unit_phase_bytes(int w, int h, int n_planes) {
  return (size_t)16 * h * unit_pitch(w) + (size_t)n_planes * sizeof(UnitPlane);
}
LUX_DEV const UnitPlane* unit_planes(const CostArgs& a) {
  return reinterpret_cast<const UnitPlane*>(reinterpret_cast<const uint8_t*>(a.phase[0]) + (size_t)16 * a.oh[0] * unit_pitch(a.ow[0]));
}

// Byte phase images: out[h][k][y][i] = phase h at column i + k - kUnitPad (clamped to the image). A thread makes four bytes of
// the four copies of every phase.
__global__ void k_phase_bytes(const uint8_t* __restrict__ img, int iw, int ih, uint8_t* __restrict__ out) {
  const int pitch = unit_pitch(iw), i4 = (blockIdx.x * blockDim.x + threadIdx.x) * 4, y = blockIdx.y;
  if (i4 >= pitch) return;
  const int y1 = min(y + 1, ih - 1);
  int r0[8], r1[8];  // columns i4 - kUnitPad .. + 7 of rows y and y + 1
#pragma unroll
  for (int c = 0; c < 8; c++) {
    const int x = min(max(i4 + c - kUnitPad, 0), iw - 1);
    r0[c] = __ldg(img + ((size_t)y * iw + x) * 4);
    r1[c] = __ldg(img + ((size_t)y1 * iw + x) * 4);
  }
#pragma unroll
  for (int h = 0; h < 4; h++) {
    int v[8];
#pragma unroll
    for (int c = 0; c < 7; c++) {
      const int a = h & 2 ? avg_u8(r0[c], r1[c]) : r0[c], b = h & 2 ? avg_u8(r0[c + 1], r1[c + 1]) : r0[c + 1];
      v[c] = h & 1 ? avg_u8(a, b) : a;
    }
#pragma unroll
    for (int k = 0; k < 4; k++)
      *reinterpret_cast<uint32_t*>(out + ((size_t)(h * 4 + k) * ih + y) * pitch + i4) =
          (uint32_t)v[k] | (uint32_t)v[k + 1] << 8 | (uint32_t)v[k + 2] << 16 | (uint32_t)v[k + 3] << 24;
  }
}

// The half-pixel target position of coordinate v of a plane (k_cost_axis's projection): w the flow-matrix factor of the axis.
LUX_DEV int unit_target(float v, float z, float zt, float inv, float w) {
  const float f = __fadd_rn(__fmul_rn(__fadd_rn(zt, __fmul_rn(__fmul_rn(v, z), w)), inv), 0.25f);
  return f2i(__fadd_rn(f, f));
}
__global__ void __launch_bounds__(256) k_unit_planes(const CostArgs a, const LayerGeom g, const float4* __restrict__ zt, UnitPlane* __restrict__ out) {
  __shared__ int s_dlo[2], s_dhi[2], s_lo[2], s_hi[2], s_cnt[2];
  const int p = blockIdx.x, t = threadIdx.x;
  const float z = g.planes[p];
  const float4 zk = zt[p];
  if (t < 2) {
    s_dlo[t] = s_lo[t] = INT_MAX;
    s_dhi[t] = INT_MIN;
    s_hi[t] = s_cnt[t] = 0;
  }
  __syncthreads();
#pragma unroll
  for (int ax = 0; ax < 2; ax++) {
    const int n = ax ? g.H : g.W, lim = (ax ? a.oh[0] : a.ow[0]) - 2;
    int lo = INT_MAX, hi = 0, cnt = 0, dlo = INT_MAX, dhi = INT_MIN;
    for (int v = t; v < n; v += 256) {
      const int q = unit_target((float)v, z, ax ? zk.y : zk.x, zk.w, ax ? a.warp[0][5] : a.warp[0][0]), iq = q >> 1;
      if (iq >= 1 && iq < lim) {
        lo = min(lo, v);
        hi = v + 1;
        cnt++;
        dlo = min(dlo, q - 2 * v);
        dhi = max(dhi, q - 2 * v);
      }
    }
    if (cnt) {
      atomicMin(&s_lo[ax], lo);
      atomicMax(&s_hi[ax], hi);
      atomicAdd(&s_cnt[ax], cnt);
      atomicMin(&s_dlo[ax], dlo);
      atomicMax(&s_dhi[ax], dhi);
    }
  }
  __syncthreads();
  if (t == 0) {
    UnitPlane u;
    const bool none = s_cnt[0] == 0 || s_cnt[1] == 0;  // nothing in the rect
    u.dx = none ? 0 : s_dlo[0];
    u.xa = none ? 0 : s_lo[0];
    u.xb = none ? 0 : s_hi[0];
    u.dy = none ? 0 : s_dlo[1];
    u.ya = none ? 0 : s_lo[1];
    u.yb = none ? 0 : s_hi[1];
    u.two_x = !none && s_dhi[0] == u.dx + 1;
    u.two_y = !none && s_dhi[1] == u.dy + 1;
    u.other = !none && (s_dhi[0] > u.dx + 1 || s_dhi[1] > u.dy + 1 || s_cnt[0] != u.xb - u.xa || s_cnt[1] != u.yb - u.ya);
    u.whole = !u.two_x && !u.two_y && !u.other;
    u.pad[0] = u.pad[1] = 0;
    out[p] = u;
  }
}

uint32_t cost_unit_norm(float norm) {
  uint8_t tab[19];
  for (int s = 0; s < 19; s++) {
    volatile float v = (float)((uint32_t)(s * 12240 + 16) >> 5) * norm;
    tab[s] = (uint8_t)(int)v;
  }
  for (uint32_t m = 0; m <= 65535 / 18; m++) {
    bool ok = true;
    for (uint32_t s = 0; s < 19 && ok; s++) ok = (s * m) >> 8 == tab[s];
    if (ok) return m;
  }
  return 0;
}

// min(|t - r|, 2) of four bytes: bit 7 of `big` says a difference of 2 or more.
LUX_DEV uint32_t capped_diff4(uint32_t t, uint32_t r) {
  const uint32_t v = __vabsdiffu4(t, r);
  const uint32_t big = ((v & 0x7e7e7e7eu) + 0x7e7e7e7eu) | v;
  const uint32_t two = (big >> 6) & 0x02020202u;
  return two | (v & ~(two >> 1) & 0x01010101u);
}

// One pixel's block at a plane by itself: its raw sum S0, or -1 where the target leaves the rect.
LUX_DEV int unit_gather(const CostArgs& a, const LayerGeom& g, const float4* __restrict__ zt, const uint8_t* bytes, int pitch, int x, int y, int p) {
  const int iw = a.ow[0], ih = a.oh[0], x1 = iw - 2, y1 = ih - 2;
  const float z = __ldg(g.planes + p), xf = (float)x, yf = (float)y;
  const float4 zk = __ldg(zt + p);
  int tx, ty;
  if (p == 0) {  // the general projection, clamped into the rect (:263-269)
    const float* Wm = a.warp[0];
    const float xz = __fmul_rn(xf, z), yz = __fmul_rn(yf, z);
    const float px = __fadd_rn(__fadd_rn(zk.x, __fmul_rn(xz, Wm[0])), __fmul_rn(yz, Wm[4]));
    const float py = __fadd_rn(__fadd_rn(zk.y, __fmul_rn(xz, Wm[1])), __fmul_rn(yz, Wm[5]));
    const float pz = __fadd_rn(__fadd_rn(zk.z, __fmul_rn(xz, Wm[2])), __fmul_rn(yz, Wm[6]));
    const float inv = __frcp_rn(pz);
    const float fx = cs_minf(cs_maxf(__fadd_rn(__fmul_rn(px, inv), 0.25f), 1.0f), (float)(x1 - 1));
    const float fy = cs_minf(cs_maxf(__fadd_rn(__fmul_rn(py, inv), 0.25f), 1.0f), (float)(y1 - 1));
    tx = f2i(__fadd_rn(fx, fx));
    ty = f2i(__fadd_rn(fy, fy));
  } else {
    tx = unit_target(xf, z, zk.x, zk.w, a.warp[0][0]);
    ty = unit_target(yf, z, zk.y, zk.w, a.warp[0][5]);
  }
  const int ix = tx >> 1, iy = ty >> 1;
  if (ix < 1 || ix >= x1 || iy < 1 || iy >= y1) return -1;
  const uint8_t* q = bytes + ((size_t)(((ty & 1) << 1) | (tx & 1)) * 4 * ih + (iy - 1)) * pitch + kUnitPad + ix - 1;
  int s = 0;
#pragma unroll
  for (int r = 0; r < 3; r++) {
    const uint8_t* rr = a.ref + (size_t)min(max(y + r - 1, 0), a.rh - 1) * a.rw * 4;
#pragma unroll
    for (int c = 0; c < 3; c++) s += min(abs((int)__ldg(q + (size_t)r * pitch + c) - (int)__ldg(rr + (size_t)min(max(x + c - 1, 0), a.rw - 1) * 4)), 2);
  }
  return s;
}

__global__ void __launch_bounds__(32) k_cost_unit(const CostArgs a, const LayerGeom g, const float4* __restrict__ zt, uint8_t* __restrict__ raw, int* err) {
  constexpr int R = kUnitRows;
  __shared__ uint32_t s_out[R][128][8];  // 32 planes of a pixel, words swizzled by the pixel
  const int lane = threadIdx.x, runs = (g.W + kUnitRun - 1) / kUnitRun, tile = blockIdx.x;
  const int n = g.n_planes, ih = a.oh[0], pitch = unit_pitch(a.ow[0]);
  const uint8_t* bytes = reinterpret_cast<const uint8_t*>(a.phase[0]);
  const UnitPlane* up = unit_planes(a);
  const int y0 = tile / runs * R, X0 = (tile % runs) * kUnitRun - 4, x0 = X0 + 4 * lane;  // columns X0..X0+127, x0: this lane's
  const bool stores = lane >= 1 && lane <= 30;
  uint32_t ref[R + 2], keep[R], last[R];
#pragma unroll
  for (int r = 0; r < R + 2; r++) {  // rows y0-1..y0+R and the columns, clamped as the reference clamps its block
    const uint8_t* row = a.ref + (size_t)min(max(y0 + r - 1, 0), a.rh - 1) * a.rw * 4;
    uint32_t w = 0;
#pragma unroll
    for (int j = 0; j < 4; j++) w |= (uint32_t)__ldg(row + (size_t)min(max(x0 + j, 0), a.rw - 1) * 4) << (8 * j);
    ref[r] = w;
  }
#pragma unroll
  for (int i = 0; i < R; i++) {  // skipped pixels' costs are 0 (DenseStereoSgm.cs:242)
    keep[i] = 0;
    last[i] = 0;
#pragma unroll
    for (int j = 0; j < 4; j++)
      if (stores && x0 + j < g.W && y0 + i < g.H && g.skip[(size_t)(y0 + i) * g.W + x0 + j] == 0) keep[i] |= 0xffu << (8 * j);
  }
  const uint32_t mul = a.norm_mul;
  auto gather = [&](int p) {  // the blocks one by one
#pragma unroll
    for (int i = 0; i < R; i++)
#pragma unroll 1
      for (int j = 0; j < 4; j++) {
        if (!((keep[i] >> (8 * j)) & 1)) continue;
        const int s = unit_gather(a, g, zt, bytes, pitch, x0 + j, y0 + i, p);
        if (s >= 0) last[i] = (last[i] & ~(0xffu << (8 * j))) | (((uint32_t)s * mul) >> 8) << (8 * j);
        else if (p == 0) atomicCAS(err, 0, 7);  // the scalar fallback of the reference would read out of the image
      }
  };
  // The costs of a plane whose block rows' capped differences are d[] (four pixels a word).
  auto sums = [&](const uint32_t (&d)[R + 2], uint32_t (&c)[R]) {
#pragma unroll
    for (int i = 0; i < R; i++) {
      const uint32_t v = d[i] + d[i + 1] + d[i + 2];
      const uint32_t left = __shfl_up_sync(0xffffffffu, v, 1), right = __shfl_down_sync(0xffffffffu, v, 1);
      const uint32_t t = v + __byte_perm(left, v, 0x6543) + __byte_perm(v, right, 0x4321);
      c[i] = __byte_perm((t & 0x00ff00ffu) * mul, ((t >> 8) & 0x00ff00ffu) * mul, 0x7351);
    }
  };
  auto plane = [&](int p) {  // makes last[] the costs of plane p
    const UnitPlane u = up[p];
    if (p == 0 || u.other) {
      gather(p);
      return;
    }
    if (u.xa >= X0 + 128 || u.xb <= X0 || u.ya >= y0 + R || u.yb <= y0) return;  // nothing in the rect: the last cost stays (:273-274)
    const float z = __ldg(g.planes + p);
    const float4 zk = __ldg(zt + p);
    uint32_t made[R];  // the costs made so far, each pixel's at its own shift
#pragma unroll
    for (int i = 0; i < R; i++) made[i] = last[i];
#pragma unroll 1
    for (int v = 0; v < 4; v++) {
      const int dx = u.dx + (v & 1), dy = u.dy + (v >> 1);
      if (((v & 1) && !u.two_x) || ((v >> 1) && !u.two_y)) continue;
      const int o = x0 + (dx >> 1) + kUnitPad;  // its low two bits are the warp's
      const uint8_t* base = bytes + (size_t)((((dy & 1) << 1) | (dx & 1)) * 4 + (o & 3)) * ih * pitch + (o & ~3);
      uint32_t d[R + 2], c[R];
#pragma unroll
      for (int r = 0; r < R + 2; r++) {
        const int row = min(max(y0 + r - 1 + (dy >> 1), 0), ih - 1);
        d[r] = capped_diff4(__ldg(reinterpret_cast<const uint32_t*>(base + (size_t)row * pitch)), ref[r]);
      }
      sums(d, c);
      uint32_t mask = 0;
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const bool mine = !u.two_x || unit_target((float)(x0 + j), z, zk.x, zk.w, a.warp[0][0]) - 2 * (x0 + j) == dx;
        if (mine && x0 + j >= u.xa && x0 + j < u.xb) mask |= 0xffu << (8 * j);
      }
#pragma unroll
      for (int i = 0; i < R; i++) {
        const int y = y0 + i;
        const bool mine = !u.two_y || unit_target((float)y, z, zk.y, zk.w, a.warp[0][5]) - 2 * y == dy;
        if (mine && y >= u.ya && y < u.yb) made[i] = (c[i] & mask) | (made[i] & ~mask);
      }
    }
#pragma unroll
    for (int i = 0; i < R; i++) last[i] = made[i];
  };
  const bool full_run = X0 + 124 <= g.W;
#pragma unroll 1
  for (int p0 = 0; p0 < n; p0 += 32) {
    const int m = min(32, n - p0);
    // lane i: plane p0 + i over this tile: all in the rect with one shift (plain), the same but for columns outside xa..xb-1
    // (partly), nothing in the rect (none), or any other (by itself); and where the tile's first block row starts
    uint32_t off = 0;
    int xa = 0, xb = 0;
    bool plain = false, partly = false, none = false;
    if (lane < m && p0 + lane > 0) {
      const UnitPlane u = up[p0 + lane];
      xa = u.xa;
      xb = u.xb;
      none = u.whole && (u.xa >= X0 + 128 || u.xb <= X0 || u.ya >= y0 + R || u.yb <= y0);
      partly = u.whole && !none && u.ya <= y0 && u.yb >= y0 + R;
      plain = partly && u.xa <= X0 && u.xb >= X0 + 128;
      const int o = X0 + (u.dx >> 1) + kUnitPad, h = ((u.dy & 1) << 1) | (u.dx & 1);
      if (partly) off = ((uint32_t)(h * 4 + (o & 3)) * ih + (uint32_t)(y0 - 1 + (u.dy >> 1))) * (uint32_t)pitch + (uint32_t)(o & ~3);
    }
    const uint32_t plain_planes = __ballot_sync(0xffffffffu, plain), none_planes = __ballot_sync(0xffffffffu, none);
    const uint32_t masked_planes = __ballot_sync(0xffffffffu, partly) | none_planes;
#pragma unroll 1
    for (int q = 0; q < m; q += 4) {
      uint32_t c[4][R];  // four planes of four pixels
      if (((none_planes >> q) & 15u) == 15u) {  // the last cost stays (:273-274)
#pragma unroll
        for (int k = 0; k < 4; k++)
#pragma unroll
          for (int i = 0; i < R; i++) c[k][i] = last[i];
      } else if (((masked_planes >> q) & 15u) == 15u) {
        uint32_t t[4][R + 2];
#pragma unroll
        for (int k = 0; k < 4; k++) {  // (planes with nothing in the rect read some words and keep none)
          const uint8_t* b = bytes + __shfl_sync(0xffffffffu, off, q + k) + 4 * lane;
#pragma unroll
          for (int r = 0; r < R + 2; r++, b += pitch) t[k][r] = __ldg(reinterpret_cast<const uint32_t*>(b));
        }
#pragma unroll
        for (int k = 0; k < 4; k++) {
#pragma unroll
          for (int r = 0; r < R + 2; r++) t[k][r] = capped_diff4(t[k][r], ref[r]);
          sums(t[k], c[k]);
        }
        if (((plain_planes >> q) & 15u) != 15u) {
#pragma unroll
          for (int k = 0; k < 4; k++) {
            int lo = min(max(__shfl_sync(0xffffffffu, xa, q + k) - x0, 0), 4), hi = min(max(__shfl_sync(0xffffffffu, xb, q + k) - x0, 0), 4);
            if ((none_planes >> (q + k)) & 1) lo = 4;
            const uint32_t mask = (lo < 4 ? 0xffffffffu << (8 * lo) : 0u) & (hi < 4 ? (1u << (8 * hi)) - 1u : 0xffffffffu);
#pragma unroll
            for (int i = 0; i < R; i++) c[k][i] = (c[k][i] & mask) | ((k ? c[k > 0 ? k - 1 : 0][i] : last[i]) & ~mask);
          }
        }
#pragma unroll
        for (int i = 0; i < R; i++) last[i] = c[3][i];
      } else {
#pragma unroll 1
        for (int k = 0; k < 4; k++) {
          plane(p0 + q + k);
#pragma unroll
          for (int i = 0; i < R; i++)
#pragma unroll
            for (int j = 0; j < 4; j++)
              reinterpret_cast<uint8_t*>(&s_out[i][j * 32 + lane][(q >> 2) ^ ((lane >> 2) & 7)])[k] = (uint8_t)((last[i] & keep[i]) >> (8 * j));
        }
        continue;
      }
#pragma unroll
      for (int i = 0; i < R; i++) {  // transposed: four planes of a pixel a word
        const uint32_t a0 = __byte_perm(c[0][i] & keep[i], c[1][i] & keep[i], 0x5140), a1 = __byte_perm(c[2][i] & keep[i], c[3][i] & keep[i], 0x5140),
                       b0 = __byte_perm(c[0][i] & keep[i], c[1][i] & keep[i], 0x7362), b1 = __byte_perm(c[2][i] & keep[i], c[3][i] & keep[i], 0x7362);
        uint32_t* o = &s_out[i][lane][(q >> 2) ^ ((lane >> 2) & 7)];
        o[0] = __byte_perm(a0, a1, 0x5410);
        o[32 * 8] = __byte_perm(a0, a1, 0x7632);
        o[64 * 8] = __byte_perm(b0, b1, 0x5410);
        o[96 * 8] = __byte_perm(b0, b1, 0x7632);
      }
    }
    __syncwarp();
    // a pixel's planes by eight lanes (32 bytes), four pixels at a time: word l, byte j of the run is pixel X0 + 4l + j
    const int w = lane & 7, sub = lane >> 3;
    if (w * 4 < m) {
#pragma unroll
      for (int i = 0; i < R; i++) {
        if (y0 + i >= g.H) break;
#pragma unroll 1
        for (int j = 0; j < 4; j++) {
          const int xj = X0 + 4 * sub + j;
          uint8_t* o = raw + ((long long)(y0 + i) * g.W + xj) * n + p0 + w * 4;
          const uint32_t* src = &s_out[i][j * 32 + sub][0];
#pragma unroll
          for (int k = 0; k < 8; k++, o += 16 * n) {
            if ((k > 0 || sub > 0) && (k < 7 || sub < 3) && (full_run || xj + 16 * k < g.W))
              *reinterpret_cast<uint32_t*>(o) = src[k * 32 + (w ^ k)];
          }
        }
      }
    }
    __syncwarp();
  }
}

bool cost_all_grey(const CostArgs& a) {
  for (int k = 0; k < a.n_others; k++)
    if (!(a.wq[k][0] == 12240 && a.wq[k][1] == 0 && a.wq[k][2] == 0 && a.wq[k][3] == 0)) return false;
  return true;
}

void launch_phases(const CostArgs& a, cudaStream_t s) {
  const bool grey = cost_all_grey(a);
  for (int k = 0; k < a.n_others; k++) {
    dim3 grid((a.ow[k] + 127) / 128, a.oh[k]);
    uint32_t* out = const_cast<uint32_t*>(a.phase[k]);
    if (a.unit)
      k_phase_bytes<<<dim3((unit_pitch(a.ow[k]) / 4 + 127) / 128, a.oh[k]), 128, 0, s>>>(a.other[k], a.ow[k], a.oh[k], reinterpret_cast<uint8_t*>(out));
    else if (a.vcols) k_phase_grey_v<<<grid, 128, 0, s>>>(a.other[k], a.ow[k], a.oh[k], reinterpret_cast<uint2*>(out));
    else if (grey) k_phase_grey<<<grid, 128, 0, s>>>(a.other[k], a.ow[k], a.oh[k], out);
    else k_phase_colour<<<grid, 128, 0, s>>>(a.other[k], a.ow[k], a.oh[k], out);
    count_launches(1);
  }
}

// The row kernels give a warp 32 pixels of a row and walk the planes in each lane: a small layer with many planes (the
// L16 pyramid's first layer: 65x49 pixels, 552 planes, 147 row tiles) leaves most SMs idle for a long walk, so it takes
// the warp-per-pixel kernel, lanes over planes (same bits), with the horizontal phase images that kernel reads.
bool cost_small_wide_layer(int W, int H, int n_planes) { return ((W + 31) / 32) * H < 148 * 4 && n_planes > 256; }

int launch_cost(const CostArgs& a, const LayerGeom& g, const float4* zt, uint8_t* raw, int* err, cudaStream_t s) {
  const int npx = g.W * g.H;
  const bool grey = cost_all_grey(a);
  int kind = 0;
  bool small_index = true;  // the row kernel's half-pixel positions are below 2^22, its offsets into phase images ints
  for (int k = 0; k < a.n_others; k++) small_index &= std::max(a.ow[k], a.oh[k]) < 1 << 20 && (size_t)a.ow[k] * a.oh[k] < (size_t)1 << 29;
  if (g.uniform && (a.axis || small_index) && !cost_small_wide_layer(g.W, g.H, g.n_planes) && g.n_planes % 8 == 0 && a.n_others >= 1 &&
      a.n_others <= kMaxCams - 1) {
    const int tiles = ((g.W + 31) / 32) * g.H;
    int blocks = (tiles + 7) / 8;
    if (blocks > 148 * 16) blocks = 148 * 16;
    if (a.unit) {
      uint8_t* ph = reinterpret_cast<uint8_t*>(const_cast<uint32_t*>(a.phase[0]));
      k_unit_planes<<<g.n_planes, 256, 0, s>>>(a, g, zt, reinterpret_cast<UnitPlane*>(ph + (size_t)16 * a.oh[0] * unit_pitch(a.ow[0])));
      count_launches(1);
      k_cost_unit<<<cost_unit_tiles(g.W, g.H), 32, 0, s>>>(a, g, zt, raw, err);
      kind = 3;
    } else if (a.vcols) {
      const int vruns = ((g.W + kAxRun - 1) / kAxRun) * g.H;
      int vb = (vruns + 7) / 8;
      if (vb > 148 * 16) vb = 148 * 16;
      k_cost_axis_v<kAxPx><<<vb, 256, 0, s>>>(a, g, zt, raw, err);
      kind = 3;
    } else if (a.axis) {
      if (grey) k_cost_axis<true><<<blocks, 256, 0, s>>>(a, g, zt, raw, err);
      else k_cost_axis<false><<<blocks, 256, 0, s>>>(a, g, zt, raw, err);
      kind = 2;
    } else {
      constexpr int kWarps = kRowsThreads / 32;
      if (grey) k_cost_rows<true><<<(tiles + kWarps - 1) / kWarps, kRowsThreads, 0, s>>>(a, g, zt, raw, err);
      else k_cost_rows<false><<<(tiles + kWarps - 1) / kWarps, kRowsThreads, 0, s>>>(a, g, zt, raw, err);
      kind = 1;
    }
  } else {
    int blocks = (npx + 7) / 8;
    if (blocks > 148 * 64) blocks = 148 * 64;
    if (grey) k_cost<true><<<blocks, 256, 0, s>>>(a, g, zt, raw, err);
    else k_cost<false><<<blocks, 256, 0, s>>>(a, g, zt, raw, err);
  }
  count_launches(1);
  return kind;
}

}  // namespace lux
