// The opt-in census stereo mode of a rectified grey pair (no counterpart in the reference, whose dense stage is the
// plane sweep): census transform, Hamming matching cost, eight-path semi-global aggregation with constant penalties P1 and
// P2, winner-take-all with parabolic subpixel refinement and a left/right consistency check, and the fusion of several
// pairs' disparities into one depth map. The method is Hirschmueller's semi-global matching (PAMI 2008) on the census
// transform of Zabih and Woodfill (ECCV 1994); the conventions (9x7 window, out-of-range cost 62, first minimum, the
// median fusion) are spelled out with each kernel.
//
// Layout in HBM: census images W x H uint64; the cost volume [pixel][Dp] uint8 and the path sums [pixel][Dp] uint16 with
// Dp = 32 x LPT >= D (LPT = 1, 2, 4 or 8). The sums that the lines leave keep lines.cuh's order within every octet.
#include <algorithm>

#include "../../include/lux_sgm.h"
#include "common.cuh"
#include "internal.h"
#include "lines.cuh"

namespace lux {

namespace {

constexpr int kCensusWX = 4, kCensusWY = 3;  // a 9x7 window: 62 bits
constexpr uint32_t kInvalidCost = 62;        // the cost where x - d leaves the image
constexpr uint32_t kBig = 1u << 20;          // disparities past D: never a minimum

// value i of a lane's LPT registers (i known only at run time)
template <int LPT>
LUX_DEV uint32_t pick(const uint32_t (&v)[LPT], int i) {
  uint32_t r = v[0];
#pragma unroll
  for (int k = 1; k < LPT; k++) r = i == k ? v[k] : r;
  return r;
}

// Disparity d of least sum b with the parabolic subpixel correction (a - c) / (2 (a - 2 b + c)), a and c the sums beside it,
// where 0 < d < D - 1 and the denominator is positive.
LUX_DEV float refine(int d, int D, int subpixel, float b, float a, float c) {
  float out = (float)d;
  if (subpixel && d > 0 && d < D - 1) {
    const float den = __fmul_rn(2.0f, __fadd_rn(__fsub_rn(a, __fmul_rn(2.0f, b)), c));
    if (den > 0.0f) out = __fadd_rn(out, __fdiv_rn(__fsub_rn(a, c), den));
  }
  return out;
}
LUX_DEV int octet_pos(int k) { return 2 * (k & 3) + (k >> 2); }  // where the lines keep plane k of an octet

// The first disparity with the least path sum S[0..D) of a pixel held by a warp (LPT a lane), refined.
template <int LPT>
LUX_DEV void wta_of(const uint32_t (&s)[LPT], int lane, int D, int subpixel, int& d_out, float& disp_out) {
  uint32_t best = kBig, arg = kBig;
#pragma unroll
  for (int i = 0; i < LPT; i++) {
    const int d = lane * LPT + i;
    const uint32_t v = d < D ? (s[i] & 0xffffu) : kBig;
    if (v < best) {
      best = v;
      arg = d;
    }
  }
  const uint32_t m = __reduce_min_sync(0xffffffffu, best);
  const int d = (int)__reduce_min_sync(0xffffffffu, best == m ? arg : kBig);
  const int dm = max(d - 1, 0), dp = min(d + 1, D - 1);
  const float a = (float)__shfl_sync(0xffffffffu, pick<LPT>(s, dm % LPT) & 0xffffu, dm / LPT);
  const float c = (float)__shfl_sync(0xffffffffu, pick<LPT>(s, dp % LPT) & 0xffffu, dp / LPT);
  d_out = d;
  disp_out = refine(d, D, subpixel, (float)m, a, c);
}

// Bit k (row-major over the window, centre skipped) is set when that neighbour, read at the clamped position, is darker
// than the centre.
__global__ void k_census(const uint8_t* __restrict__ img, int w, int h, int stride, int bpp, uint64_t* __restrict__ out) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
  if (x >= w || y >= h) return;
  auto at = [&](int xx, int yy) { return (int)__ldg(img + ((size_t)min(max(yy, 0), h - 1) * stride + min(max(xx, 0), w - 1)) * bpp); };
  const int c = at(x, y);
  uint64_t v = 0;
  int bit = 0;
#pragma unroll
  for (int dy = -kCensusWY; dy <= kCensusWY; dy++)
#pragma unroll
    for (int dx = -kCensusWX; dx <= kCensusWX; dx++) {
      if (dx == 0 && dy == 0) continue;
      v |= (uint64_t)(at(x + dx, y + dy) < c) << bit;
      bit++;
    }
  out[(size_t)y * w + x] = v;
}

// C(x, y, d) = popcount(L(x, y) ^ R(x - d, y)), 62 where x - d < 0. A block takes kHamTile pixels of a row, a thread eight
// disparities of a pixel at a time, stored as one word pair; the right image's words wait in shared memory, their halves apart
// and a word skipped every eight, so that threads eight words apart meet no bank twice. Bound by the population counts (16 a
// clock an SM): 2080x1560 D=128 in 273 us; a warp a pixel storing bytes took 418, this from global memory 769.
constexpr int kHamTile = 64;
template <int LPT>
__global__ void __launch_bounds__(256) k_hamming(const uint64_t* __restrict__ cl, const CensusPairs ps, int w, int h, int tiles) {
  constexpr int Dp = 32 * LPT, GL = 4 * LPT, kWords = kHamTile + Dp - 1;  // GL: threads of a pixel
  __shared__ uint32_t lo[kWords + kWords / 8 + 1], hi[kWords + kWords / 8 + 1];
  const CensusPair& pr = ps.p[blockIdx.y];  // one grid row per pair of the batch
  const int y = blockIdx.x / tiles, x0 = (blockIdx.x - y * tiles) * kHamTile, D = pr.D;
  for (int i = threadIdx.x; i < kWords; i += 256) {  // word i: R(x0 - (Dp - 1) + i, y)
    const int xr = x0 - (Dp - 1) + i;
    const uint64_t v = xr >= 0 && xr < w ? __ldg(pr.cr + (size_t)y * w + xr) : 0;
    lo[i + i / 8] = (uint32_t)v;
    hi[i + i / 8] = (uint32_t)(v >> 32);
  }
  __syncthreads();
  for (int t = threadIdx.x; t < kHamTile * GL; t += 256) {
    const int x = x0 + t / GL, d0 = (t % GL) * 8;
    if (x >= w) break;
    const size_t p = (size_t)y * w + x;
    const uint64_t a = __ldg(cl + p);
    const uint32_t al = (uint32_t)a, ah = (uint32_t)(a >> 32);
    const int r = t / GL + Dp - 1 - d0, live = min(D - d0, x - d0 + 1);  // the word of d0; how many of the disparities count
    uint32_t c[8];
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const int j = r - i + (r - i) / 8;
      c[i] = __popc(al ^ lo[j]) + __popc(ah ^ hi[j]);
    }
    if (live < 8) {
#pragma unroll
      for (int i = 0; i < 8; i++) c[i] = i < live ? c[i] : kInvalidCost;
    }
    reinterpret_cast<uint2*>(pr.cost + p * Dp)[t % GL] =
        make_uint2(c[0] | c[1] << 8 | c[2] << 16 | c[3] << 24, c[4] | c[5] << 8 | c[6] << 16 | c[7] << 24);
  }
}

// A lane's LPT cost bytes and LPT path sums as one vector access each.
template <int LPT>
struct LaneIO;
template <>
struct LaneIO<1> {
  static LUX_DEV void cost(const uint8_t* p, uint32_t (&c)[1]) { c[0] = *p; }
  static LUX_DEV void load(const uint16_t* p, uint32_t (&v)[1]) { v[0] = *p; }
  static LUX_DEV void store(uint16_t* p, const uint32_t (&v)[1]) { *p = (uint16_t)v[0]; }
};
template <>
struct LaneIO<2> {
  static LUX_DEV void cost(const uint8_t* p, uint32_t (&c)[2]) {
    const uint32_t w = *reinterpret_cast<const uint16_t*>(p);
    c[0] = w & 0xff;
    c[1] = w >> 8;
  }
  static LUX_DEV void load(const uint16_t* p, uint32_t (&v)[2]) {
    const uint32_t w = *reinterpret_cast<const uint32_t*>(p);
    v[0] = w & 0xffff;
    v[1] = w >> 16;
  }
  static LUX_DEV void store(uint16_t* p, const uint32_t (&v)[2]) { *reinterpret_cast<uint32_t*>(p) = v[0] | v[1] << 16; }
};
template <>
struct LaneIO<4> {
  static LUX_DEV void cost(const uint8_t* p, uint32_t (&c)[4]) {
    const uint32_t w = *reinterpret_cast<const uint32_t*>(p);
#pragma unroll
    for (int i = 0; i < 4; i++) c[i] = (w >> (8 * i)) & 0xff;
  }
  static LUX_DEV void load(const uint16_t* p, uint32_t (&v)[4]) {
    const uint2 w = *reinterpret_cast<const uint2*>(p);
    v[0] = w.x & 0xffff;
    v[1] = w.x >> 16;
    v[2] = w.y & 0xffff;
    v[3] = w.y >> 16;
  }
  static LUX_DEV void store(uint16_t* p, const uint32_t (&v)[4]) {
    *reinterpret_cast<uint2*>(p) = make_uint2(v[0] | v[1] << 16, v[2] | v[3] << 16);
  }
};
template <>
struct LaneIO<8> {
  static LUX_DEV void cost(const uint8_t* p, uint32_t (&c)[8]) {
    const uint2 w = *reinterpret_cast<const uint2*>(p);
#pragma unroll
    for (int i = 0; i < 4; i++) {
      c[i] = (w.x >> (8 * i)) & 0xff;
      c[4 + i] = (w.y >> (8 * i)) & 0xff;
    }
  }
  static LUX_DEV void load(const uint16_t* p, uint32_t (&v)[8]) {
    const uint4 w = *reinterpret_cast<const uint4*>(p);
    const uint32_t ws[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int i = 0; i < 4; i++) {
      v[2 * i] = ws[i] & 0xffff;
      v[2 * i + 1] = ws[i] >> 16;
    }
  }
  static LUX_DEV void store(uint16_t* p, const uint32_t (&v)[8]) {
    *reinterpret_cast<uint4*>(p) = make_uint4(v[0] | v[1] << 16, v[2] | v[3] << 16, v[4] | v[5] << 16, v[6] | v[7] << 16);
  }
};

// One warp walks one scanline of direction (dx, dy):
//   L(p, d) = C(p, d) + min(L(q, d), L(q, d - 1) + P1, L(q, d + 1) + P1, m + P2) - m,  m = min_k L(q, k),
// with q the previous pixel (L = C at the first pixel), and adds L into the path sums (the first direction stores them).
// The scanline starts are the pixels whose previous pixel lies outside the image: a whole row for dy != 0, then a whole
// column (less the corner already counted) for dx != 0. The next pixel's cost and sums are loaded while this one is
// computed, so the HBM latency is off the recurrence.
template <int LPT, bool LAST>
__global__ void __launch_bounds__(128) k_census_path(const CensusPairs ps, int w, int h, int dx, int dy, uint32_t P1, uint32_t P2,
                                                     int first, int subpixel) {
  constexpr int Dp = 32 * LPT;
  const CensusPair& pr = ps.p[blockIdx.y];  // one grid row per pair of the batch
  const uint8_t* __restrict__ cost = pr.cost;
  uint16_t* __restrict__ S = pr.S;
  int* __restrict__ dl = pr.dl;
  float* __restrict__ disp = pr.disp;
  const int D = pr.D;
  using IO = LaneIO<LPT>;
  const int lane = threadIdx.x & 31;
  const int line = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int n_row = dy != 0 ? w : 0, n_col = dx != 0 ? h - (dy != 0 ? 1 : 0) : 0;
  if (line >= n_row + n_col) return;
  int x, y;
  if (line < n_row) {
    x = line;
    y = dy > 0 ? 0 : h - 1;
  } else {
    x = dx > 0 ? 0 : w - 1;
    const int k = line - n_row;
    y = dy == 0 ? k : (dy > 0 ? k + 1 : k);  // the corner row was started by the row starts
  }
  auto at = [&](int xx, int yy) { return ((size_t)yy * w + xx) * Dp + lane * LPT; };
  uint32_t L[LPT], c[LPT], sv[LPT];
  uint32_t m = 0;
  IO::cost(cost + at(x, y), c);
  if (!first) IO::load(S + at(x, y), sv);
  bool start = true;
  for (;;) {
    const int xn = x + dx, yn = y + dy;
    const bool more = xn >= 0 && xn < w && yn >= 0 && yn < h;
    uint32_t cn[LPT], sn[LPT];
    if (more) {
      IO::cost(cost + at(xn, yn), cn);
      if (!first) IO::load(S + at(xn, yn), sn);
    }
    uint32_t nl[LPT];
    if (start) {
#pragma unroll
      for (int i = 0; i < LPT; i++) nl[i] = lane * LPT + i < D ? c[i] : kBig;
      start = false;
    } else {
      const uint32_t left = __shfl_up_sync(0xffffffffu, L[LPT - 1], 1), right = __shfl_down_sync(0xffffffffu, L[0], 1);
#pragma unroll
      for (int i = 0; i < LPT; i++) {
        const uint32_t lm = i > 0 ? L[i - 1] : (lane > 0 ? left : kBig);
        const uint32_t lp = i < LPT - 1 ? L[i + 1] : (lane < 31 ? right : kBig);
        const uint32_t t = min(min(L[i], min(lm, lp) + P1), m + P2);
        nl[i] = lane * LPT + i < D ? c[i] + t - m : kBig;
      }
    }
    uint32_t lmin = kBig, out[LPT];
#pragma unroll
    for (int i = 0; i < LPT; i++) {
      L[i] = nl[i];
      lmin = min(lmin, nl[i]);
      out[i] = first ? nl[i] : sv[i] + nl[i];  // padding lanes store don't-care values (never read)
    }
    m = __reduce_min_sync(0xffffffffu, lmin);
    IO::store(S + at(x, y), out);
    if (LAST) {  // the path sums of this pixel are final: the winner-take-all here saves reading them again
      int d;
      float v;
      wta_of<LPT>(out, lane, D, subpixel, d, v);
      if (lane == 0) {
        dl[(size_t)y * w + x] = d;
        disp[(size_t)y * w + x] = v;
      }
    }
    if (!more) break;
    x = xn;
    y = yn;
#pragma unroll
    for (int i = 0; i < LPT; i++) {
      c[i] = cn[i];
      sv[i] = sn[i];
    }
  }
}

// The paths along single lines, as k_lines_walk of sgm_lines.cu walks them, without its revisits and with constant penalties:
// a lane holds eight disparities as u16 pairs, a line takes GL = Dp / 8 lanes, the forward states are kept every kSeg pixels
// and the pair walk of a path shares its launch with the forward walk of the next. A line starts from L = 0 (its first step
// is then L = C). Disparities past D cost kBeyond more than their byte: they stay above every true L (62 + P2 <= 8191), and
// above m + P2 also as neighbours. Their sums may wrap: the high half of a pair never carries into a true one (plane p + 4
// is past D where plane p is), and the winner-take-all takes them as 0xffff (eight true L sum up to 65528 at most).
// The eight walks of one disparity a lane, one warp a line and one pixel of prefetch took 10.4 ms at 2080x1560 D=128 (each
// was bound by its steps' latency, at 1.2 TB/s); these take 3.0 ms.
constexpr uint32_t kBeyond = 0x40004000u;

struct CensusLines {
  int W, H, n;  // n: Dp
  uint32_t p1x2, p2x2, one;
  int subpixel, keep;  // keep: the sums are read again
  uint16_t *ckpt, *ckpt_min;  // per pair of the launch [2][states][n] and [2][states], even and odd paths
  size_t states;
  CensusPairs ps;
};

// unpack with the disparities past D raised by kBeyond
LUX_DEV void unpack_cost(L4& v, uint2 b, const L4& pad) {
  unpack(v, b);
#pragma unroll
  for (int k = 0; k < 4; k++) v.r[k] |= pad.r[k];
}
LUX_DEV L4 pad_of(int gl, int D, uint32_t value) {
  L4 v;
#pragma unroll
  for (int k = 0; k < 4; k++)
    v.r[k] = (gl * 8 + k >= D ? value & 0xffffu : 0u) | (gl * 8 + k + 4 >= D ? value & 0xffff0000u : 0u);
  return v;
}
LUX_DEV void set_zero(L4& v, uint32_t& md) { v.r[0] = v.r[1] = v.r[2] = v.r[3] = md = 0; }

template <int GL, int P>
LUX_DEV void census_forward(const CensusLines& a, const CensusPair& pr, int wi, uint2* ring, uint16_t* ckpt, uint16_t* ckpt_min) {
  constexpr int LPW = 32 / GL;
  static_assert(kBatch == kSeg, "one state a batch");
  const int n = a.n, lane = threadIdx.x & 31, gl = lane & (GL - 1), grp = lane / GL;
  const int NL = line_count(a, P);
  if (wi * LPW >= NL) return;
  const int line0 = wi * LPW + grp, line = min(line0, NL - 1);
  const bool in = line0 < NL, first = gl == 0, last = gl == GL - 1;
  const int NS = line_len(a, P, line);
  Walk w = walk_at(a, P, line_first(a, P, line), 1), ws = w;
  const L4 pad = pad_of(gl, pr.D, kBeyond);
  RawRing<8> rr(ring + lane, in);
  L4 L;
  uint32_t md;
  set_zero(L, md);
  const int steps = __reduce_max_sync(0xffffffffu, NS), nb = (steps + kBatch - 1) / kBatch;
  stage_batch(rr, 0, pr.cost, n, ws, NS, gl, in);
  ws.advance();
  stage_batch(rr, 1, pr.cost, n, ws, NS - kBatch, gl, in);
  ws.advance();
  for (int b = 0; b + 1 < nb; b++) {  // (no state is kept after the last batch)
    cp_async_wait<1>();
    bool odd = (b + 1) * kBatch > NS;  // else a whole batch without a new line
    if (P == 1) odd |= w.x == 0 || w.x + kBatch > a.W;
    if (P == 3) odd |= w.x == a.W - 1 || w.x + 1 < kBatch;
    if (!__any_sync(0xffffffffu, odd)) {
      uint2 rb[kBatch];
#pragma unroll
      for (int i = 0; i < kBatch; i++) rb[i] = rr.get(b, i);
#pragma unroll
      for (int i = 0; i < kBatch; i++) {
        L4 raw2;
        unpack_cost(raw2, rb[i], pad);
        line_step<GL, kBeyond>(L, md, raw2, a.p2x2, a, first, last);
      }
    } else {
      int x = w.x;
#pragma unroll 1
      for (int i = 0; i < kBatch; i++) {
        if ((P == 1 && x == 0) || (P == 3 && x == a.W - 1)) set_zero(L, md);
        L4 raw2;
        unpack_cost(raw2, rr.get(b, i), pad);
        line_step<GL, kBeyond>(L, md, raw2, a.p2x2, a, first, last);
        x += w.dx;
        if ((unsigned)x >= (unsigned)a.W) x -= w.dx * a.W;
      }
    }
    if (in && (b + 1) * kSeg < NS) {
      const size_t ci = (size_t)b * NL + line;
      __stcs(reinterpret_cast<uint4*>(ckpt + ci * n) + gl, as_uint4(L));
      if (gl == 0) ckpt_min[ci] = (uint16_t)(md & 0xffffu);
    }
    w.advance();
    stage_batch(rr, b + 2, pr.cost, n, ws, NS - (b + 2) * kBatch, gl, in);
    ws.advance();
  }
  cp_async_wait<0>();
}

// MODE 0 stores the sums, 1 adds to them, 2 adds, stores them where they are kept, and takes the winner.
template <int GL, int P, int MODE>
LUX_DEV void census_pair(const CensusLines& a, const CensusPair& pr, int wi, uint4* sum, uint2* rawp, const uint16_t* ckpt,
                         const uint16_t* ckpt_min) {
  constexpr int LPW = 32 / GL, dx = P == 1 ? 1 : P == 3 ? -1 : 0, PX = GL < kSeg ? kSeg / GL : 1;  // PX: a segment's pixels a lane
  const int W = a.W, n = a.n, lane = threadIdx.x & 31, gl = lane & (GL - 1), grp = lane / GL;
  const int NL = line_count(a, P);
  if (wi * LPW >= NL) return;
  const int line0 = wi * LPW + grp, line = min(line0, NL - 1);
  const bool in = line0 < NL, first = gl == 0, last = gl == GL - 1;
  const int NS = line_len(a, P, line), step = line_step_of(P, W);
  const int steps = __reduce_max_sync(0xffffffffu, NS), nseg = (steps + kSeg - 1) / kSeg;
  const L4 pad = pad_of(gl, pr.D, kBeyond);
  sum += lane;
  rawp += lane;
  if (!in)
    for (int i = 0; i < kSeg; i++) rawp[i * 32] = kPastRaw;
  int pi0 = line_first(a, P, line) + (nseg - 1) * kSeg * step, x0 = dx != 0 ? pi0 % W : 0;  // of the segment in hand
  auto stage = [&](int i, int pi) {
    if (MODE != 0) cp_async16(sum + i * 32, reinterpret_cast<const uint4*>(pr.S + (size_t)pi * n) + gl);
    cp_async8(rawp + i * 32, reinterpret_cast<const uint2*>(pr.cost + (size_t)pi * n) + gl);
  };
  for (int i = 0; i < kSeg; i++)
    if (in && (nseg - 1) * kSeg + i < NS) stage(i, pi0 + step * i);
  cp_async_commit();
  auto load_ckpt = [&](int seg, L4& L, uint32_t& mn) {  // the forward state before segment seg, its minimum not yet doubled
    set_zero(L, mn);
    if (seg > 0 && seg * kSeg < NS && in) {
      const size_t ci = (size_t)(seg - 1) * NL + line;
      L = as_l4(__ldcs(reinterpret_cast<const uint4*>(ckpt + ci * n) + gl));
      mn = __ldcs(ckpt_min + ci);
    }
  };
  L4 F, B;  // the forward and backward states
  uint32_t fd, bd;
  load_ckpt(nseg - 1, F, fd);
  fd = dup16(fd);
  set_zero(B, bd);
  for (int seg = nseg - 1; seg >= 0; seg--) {
    const int t0 = seg * kSeg;
    cp_async_wait<0>();
    // a whole segment clear of new lines either way (where two lines of a warp end a step apart, one of
    // them is at a side in the segment in which the shorter one ends)
    bool odd = t0 + kSeg > NS;
    if (P == 1) odd |= x0 == 0 || x0 + kSeg >= W;
    if (P == 3) odd |= x0 == W - 1 || x0 < kSeg;
    const bool plain = seg > 0 && !__any_sync(0xffffffffu, odd);
    auto add_fwd = [&](int i) {
      if (MODE == 0) {
        sum[i * 32] = as_uint4(F);
      } else {
        uint4 s = sum[i * 32];
        s.x += F.r[0];
        s.y += F.r[1];
        s.z += F.r[2];
        s.w += F.r[3];
        sum[i * 32] = s;
      }
    };
    if (plain) {
#pragma unroll
      for (int i = 0; i < kSeg; i++) {
        L4 raw2;
        unpack_cost(raw2, rawp[i * 32], pad);
        line_step<GL, kBeyond>(F, fd, raw2, a.p2x2, a, first, last);
        add_fwd(i);
      }
    } else {
      int x = x0;
#pragma unroll 1
      for (int i = 0; i < kSeg; i++) {
        if ((P == 1 && x == 0) || (P == 3 && x == W - 1)) set_zero(F, fd);
        L4 raw2;
        unpack_cost(raw2, rawp[i * 32], pad);
        line_step<GL, kBeyond>(F, fd, raw2, a.p2x2, a, first, last);
        add_fwd(i);
        x += dx;
        if ((unsigned)x >= (unsigned)W) x -= dx * W;
      }
    }
    const int pq = pi0 - step * kSeg;  // the segment before
    L4 Fn;
    uint32_t fdn;
    load_ckpt(seg - 1, Fn, fdn);
    // lane i (mod GL): the segment's pixels i, i + GL: the winner, its sum, and the sums beside it (low and high half)
    int win[PX] = {};
    uint32_t least[PX] = {}, beside[PX] = {};
    auto put = [&](int i, int pi, bool live) {
      L4 s = as_l4(sum[i * 32]);
#pragma unroll
      for (int k = 0; k < 4; k++) s.r[k] += B.r[k];
      if ((MODE != 2 || a.keep) && in && live) __stcs(reinterpret_cast<uint4*>(pr.S + (size_t)pi * n) + gl, as_uint4(s));
      if constexpr (MODE == 2) {
        const L4 full = pad_of(gl, pr.D, 0xffffffffu);
#pragma unroll
        for (int k = 0; k < 4; k++) s.r[k] |= full.r[k];
        const int arg = wta_line<GL>(s, gl, lane, true);
        sum[i * 32] = as_uint4(s);
        __syncwarp();
        const uint16_t* sums = reinterpret_cast<const uint16_t*>(sum + i * 32 - gl);
        auto at = [&](int d) { return (uint32_t)sums[(d & ~7) + octet_pos(d & 7)]; };
        if ((gl & (kSeg - 1)) == (i & (GL - 1) & (kSeg - 1))) {
          const uint32_t m = at(arg), bs = at(max(arg - 1, 0)) | at(min(arg + 1, pr.D - 1)) << 16;
#pragma unroll
          for (int k = 0; k < PX; k++)
            if (k == i / GL) {
              win[k] = arg;
              least[k] = m;
              beside[k] = bs;
            }
        }
        __syncwarp();
      }
    };
    if (plain) {
#pragma unroll
      for (int i = kSeg - 1; i >= 0; i--) {
        L4 raw2;
        unpack_cost(raw2, rawp[i * 32], pad);
        line_step<GL, kBeyond>(B, bd, raw2, a.p2x2, a, first, last);
        put(i, pi0 + step * i, true);
        if (in) stage(i, pq + step * i);
      }
    } else {
      int x = x0 + dx * (kSeg - 1), pi = pi0 + step * (kSeg - 1);
      if ((unsigned)x >= (unsigned)W) x -= dx * W;
#pragma unroll 1
      for (int i = kSeg - 1; i >= 0; i--) {
        // the line's last pixel, or a new line: the way back comes in at the side the diagonal left by
        if (t0 + i == NS - 1 || (P == 1 && x == W - 1) || (P == 3 && x == 0)) set_zero(B, bd);
        L4 raw2;
        unpack_cost(raw2, rawp[i * 32], pad);
        line_step<GL, kBeyond>(B, bd, raw2, a.p2x2, a, first, last);
        put(i, pi, t0 + i < NS);
        if (seg > 0 && in && t0 - kSeg + i < NS) stage(i, pq + step * i);
        pi -= step;
        x -= dx;
        if ((unsigned)x >= (unsigned)W) x += dx * W;
      }
    }
    cp_async_commit();
    if (MODE == 2 && gl < kSeg) {
#pragma unroll
      for (int k = 0; k < PX; k++) {
        const int i = gl + k * GL;
        if (in && t0 + i < NS) {
          pr.dl[pi0 + step * i] = win[k];
          pr.disp[pi0 + step * i] = refine(win[k], pr.D, a.subpixel, (float)least[k], (float)(beside[k] & 0xffffu), (float)(beside[k] >> 16));
        }
      }
    }
    F = Fn;
    fd = dup16(fdn);
    pi0 = pq;
    x0 -= dx * kSeg;
    if ((unsigned)x0 >= (unsigned)W) x0 += dx * W;
  }
}

// The pair walk of path P (its warps first) beside the forward walk of path NEXT; -1: none. A grid row a pair of images.
template <int GL, int P, int MODE, int NEXT>
__global__ void __launch_bounds__(64, 16) k_census_walk(const __grid_constant__ CensusLines a) {
  constexpr int LPW = 32 / GL, PP = P < 0 ? 0 : P, PN = NEXT < 0 ? 0 : NEXT;
  __shared__ uint4 s_sum[2][kSeg * 32];
  __shared__ uint2 s_raw[2][kSeg * 32];
  const int wib = threadIdx.x >> 5;
  const CensusPair& pr = a.ps.p[blockIdx.y];
  uint16_t* ckpt[2];
  uint16_t* ckpt_min[2];
  for (int k = 0; k < 2; k++) {
    ckpt[k] = a.ckpt + (blockIdx.y * 2 + k) * a.states * a.n;
    ckpt_min[k] = a.ckpt_min + (blockIdx.y * 2 + k) * a.states;
  }
  const int pair_blocks = P < 0 ? 0 : ((line_count(a, PP) + LPW - 1) / LPW + 1) / 2, block = blockIdx.x;
  if (P >= 0 && block < pair_blocks) {
    census_pair<GL, PP, MODE>(a, pr, block * 2 + wib, s_sum[wib], s_raw[wib], ckpt[PP & 1], ckpt_min[PP & 1]);
  } else if (NEXT >= 0) {
    census_forward<GL, PN>(a, pr, (block - pair_blocks) * 2 + wib, reinterpret_cast<uint2*>(s_sum[wib]), ckpt[PN & 1], ckpt_min[PN & 1]);
  }
}

template <int GL, int P, int MODE, int NEXT>
void run_census_walk(const CensusLines& a, int n, cudaStream_t s) {
  constexpr int LPW = 32 / GL;
  auto blocks_of = [&](int p) {
    const int lines = p < 0 ? 0 : p == 0 ? a.H : p == 1 ? a.W + 1 : p == 2 ? a.W : a.W - 1;
    return ((lines + LPW - 1) / LPW + 1) / 2;
  };
  k_census_walk<GL, P, MODE, NEXT><<<dim3(blocks_of(P) + blocks_of(NEXT), n), 64, 0, s>>>(a);
}

// The right image's first minimum over d of S(x + d, y, d), x + d < W. A block takes kRight right pixels of a row, a thread each,
// sixteen disparities at a time: their sums of the kRight + 15 left pixels they meet (a sector of each) go through shared
// memory, nine words apart so that a warp's diagonal reads meet no bank twice. Bound by HBM: 2080x1560 D=128 in 231 us; a
// warp a right pixel, reading its sums where they lay, took 580. OCTETS: the sums are in the lines' order.
constexpr int kRight = 128;
template <int LPT, bool OCTETS>
__global__ void __launch_bounds__(kRight) k_census_wta_right(const CensusPairs ps, int w, int h, int tiles) {
  constexpr int Dp = 32 * LPT, kWide = kRight + 15;
  __shared__ uint32_t sums[2][kWide * 9];
  const CensusPair& pr = ps.p[blockIdx.y];
  const int y = blockIdx.x / tiles, x0 = (blockIdx.x - y * tiles) * kRight, x = x0 + threadIdx.x;
  const uint16_t* row = pr.S + (size_t)y * w * Dp;
  uint32_t best = ~0u;  // the sum, then the disparity
  const int chunks = min((pr.D + 15) / 16, (w - x0 + 15) / 16);
  for (int c = 0; c < chunks; c++) {
    uint32_t* buf = sums[c & 1];  // (a thread is at most one chunk ahead of another)
    const int xa = x0 + c * 16;
    for (int i = threadIdx.x; i < kWide * 2; i += kRight) {
      const int px = i >> 1, hf = i & 1;
      if (xa + px >= w) break;
      const uint4 v = __ldcs(reinterpret_cast<const uint4*>(row + (size_t)(xa + px) * Dp + c * 16) + hf);
      uint32_t* q = buf + px * 9 + hf * 4;
      q[0] = v.x;
      q[1] = v.y;
      q[2] = v.z;
      q[3] = v.w;
    }
    __syncthreads();
    const uint16_t* mine = reinterpret_cast<const uint16_t*>(buf + threadIdx.x * 9);
#pragma unroll
    for (int i = 0; i < 16; i++) {
      const int d = c * 16 + i;
      const uint32_t v = mine[i * 18 + (OCTETS ? (i & 8) + octet_pos(i & 7) : i)];
      if (d < pr.D && x + d < w) best = min(best, v << 8 | (uint32_t)d);
    }
  }
  if (x < w) pr.dr[(size_t)y * w + x] = (int)(best & 0xffu);
}

// Left/right consistency: a pixel keeps its disparity when |d(x) - d_R(x - d(x))| <= max_diff, else -1.
__global__ void k_census_lr(const CensusPairs ps, int w, int h, int max_diff) {
  const CensusPair& pr = ps.p[blockIdx.y];
  const int* __restrict__ dl = pr.dl;
  const int* __restrict__ dr = pr.dr;
  float* __restrict__ disp = pr.disp;
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= w * h) return;
  const int y = p / w, x = p - y * w, d = dl[p], xr = x - d;
  if (xr < 0 || abs(d - dr[(size_t)y * w + xr]) > max_diff) disp[p] = -1.0f;
}

// The median of a pixel's valid depths fB_k / d_k (d_k > 0) over the pairs (the mean of the two middle ones for an even
// count), 0 where none is valid.
__global__ void k_fuse(const float* const* __restrict__ disps, const float* __restrict__ fb, int n, int npx, float* __restrict__ out) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= npx) return;
  float z[kMaxFusePairs];
  int k = 0;
  for (int i = 0; i < n; i++) {
    const float d = disps[i][p];
    if (d > 0.0f) {
      const float v = __fdiv_rn(fb[i], d);
      int j = k++;
      while (j > 0 && z[j - 1] > v) {  // insertion, ascending
        z[j] = z[j - 1];
        j--;
      }
      z[j] = v;
    }
  }
  out[p] = k == 0 ? 0.0f : (k & 1) ? z[k / 2] : __fmul_rn(__fadd_rn(z[k / 2 - 1], z[k / 2]), 0.5f);
}

template <int LPT>
void batch_stages(const uint64_t* cl, const CensusPairs& ps, int n, int w, int h, uint32_t P1, uint32_t P2, int subpixel, int lr,
                  int max_diff, const CensusScratch& sc, cudaStream_t s) {
  const int npx = w * h;
  constexpr int GL = 4 * LPT;
  const int tiles_h = (w + kHamTile - 1) / kHamTile;
  k_hamming<LPT><<<dim3((unsigned)tiles_h * h, n), 256, 0, s>>>(cl, ps, w, h, tiles_h);
  count_launches(1);
  const bool lines = sc.ckpt && census_lines_supported(w, h, 32 * LPT);
  if (lines) {
    CensusLines a{};
    a.W = w;
    a.H = h;
    a.n = 32 * LPT;
    a.p1x2 = P1 * 0x10001u;
    a.p2x2 = P2 * 0x10001u;
    a.one = 1;
    a.subpixel = subpixel;
    a.keep = lr;
    a.states = census_states(w, h);
    a.ckpt = sc.ckpt;
    a.ckpt_min = sc.ckpt_min;
    for (int k0 = 0; k0 < n; k0 += sc.pairs) {
      const int m = std::min(sc.pairs, n - k0);
      for (int k = 0; k < m; k++) a.ps.p[k] = ps.p[k0 + k];
      run_census_walk<GL, -1, 0, 0>(a, m, s);
      run_census_walk<GL, 0, 0, 1>(a, m, s);
      run_census_walk<GL, 1, 1, 2>(a, m, s);
      run_census_walk<GL, 2, 1, 3>(a, m, s);
      run_census_walk<GL, 3, 2, -1>(a, m, s);
      count_launches(5);
    }
  } else {
    static const int dirs[8][2] = {{1, 0}, {-1, 0}, {0, 1}, {0, -1}, {1, 1}, {-1, -1}, {1, -1}, {-1, 1}};
    for (int k = 0; k < 8; k++) {
      const int dx = dirs[k][0], dy = dirs[k][1];
      const int lines = (dy != 0 ? w : 0) + (dx != 0 ? h - (dy != 0 ? 1 : 0) : 0);
      const dim3 grid((lines + 3) / 4, n);
      if (k == 7) k_census_path<LPT, true><<<grid, 128, 0, s>>>(ps, w, h, dx, dy, P1, P2, 0, subpixel);
      else k_census_path<LPT, false><<<grid, 128, 0, s>>>(ps, w, h, dx, dy, P1, P2, k == 0 ? 1 : 0, subpixel);
    }
    count_launches(8);
  }
  if (lr) {
    const int tiles = (w + kRight - 1) / kRight;
    const dim3 right((unsigned)tiles * h, n);
    if (lines) k_census_wta_right<LPT, true><<<right, kRight, 0, s>>>(ps, w, h, tiles);
    else k_census_wta_right<LPT, false><<<right, kRight, 0, s>>>(ps, w, h, tiles);
    k_census_lr<<<dim3((npx + 255) / 256, n), 256, 0, s>>>(ps, w, h, max_diff);
    count_launches(2);
  }
}

}  // namespace

// The states of the longest walk of a pair: W + 1 lines or fewer of at most H + H / (W - 1) + 1 steps, or H lines of W.
size_t census_states(int w, int h) {
  return std::max((size_t)(w + 1) * ((h + h / (w - 1) + 1) / kSeg + 1), (size_t)h * (w / kSeg + 1));
}
// The lines walk each path but the first down the whole image, whatever its width; a scanline of a diagonal is as short as
// the shorter side. Tall images of few columns have too few lines to hide that (ms, lines / scanlines: D=64 16x2000 2.8 / 1.6,
// 64x1000 1.5 / 1.2, 100x1000 1.8 / 1.6, 200x800 1.8 / 1.8, 400x1000 3.1 / 3.7; past 64 disparities 64x5000 D=128 6.9 / 7.8,
// 16x2000 D=256 2.3 / 1.9).
bool census_lines_supported(int w, int h, int D) { return w >= kBatch && h <= (D <= 64 ? 3 : 80) * (long long)w; }
int census_lpt(int D) { return D <= 32 ? 1 : D <= 64 ? 2 : D <= 128 ? 4 : D <= 256 ? 8 : 0; }

void launch_census_batch(const uint8_t* ref, const uint8_t* const* others, int n, int w, int h, int stride, int bpp, uint32_t P1,
                         uint32_t P2, int subpixel, int lr, int max_diff, uint64_t* cl, const CensusPairs& ps, const CensusScratch& sc, cudaStream_t s) {
  const dim3 b2(32, 8), g2((w + 31) / 32, (h + 7) / 8);
  k_census<<<g2, b2, 0, s>>>(ref, w, h, stride, bpp, cl);  // the reference's census, shared by every pair
  for (int k = 0; k < n; k++) k_census<<<g2, b2, 0, s>>>(others[k], w, h, stride, bpp, ps.p[k].cr);
  count_launches(1 + n);
  // the pairs grouped by lane width (disparities a lane), one launch per stage and group
  for (const int lpt : {1, 2, 4, 8}) {
    CensusPairs grp{};
    int m = 0;
    for (int k = 0; k < n; k++)
      if (census_lpt(ps.p[k].D) == lpt) grp.p[m++] = ps.p[k];
    if (m == 0) continue;
    switch (lpt) {
      case 1: batch_stages<1>(cl, grp, m, w, h, P1, P2, subpixel, lr, max_diff, sc, s); break;
      case 2: batch_stages<2>(cl, grp, m, w, h, P1, P2, subpixel, lr, max_diff, sc, s); break;
      case 4: batch_stages<4>(cl, grp, m, w, h, P1, P2, subpixel, lr, max_diff, sc, s); break;
      default: batch_stages<8>(cl, grp, m, w, h, P1, P2, subpixel, lr, max_diff, sc, s); break;
    }
  }
}

void launch_fuse(const float* const* disps, const float* fb, int n, int npx, float* out, cudaStream_t s) {
  k_fuse<<<(npx + 255) / 256, 256, 0, s>>>(disps, fb, n, npx, out);
  count_launches(1);
}

}  // namespace lux
