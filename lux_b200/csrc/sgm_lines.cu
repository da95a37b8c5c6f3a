// Aggregation of a uniform layer by single lines (bit-exact with DenseStereoSgm.cs:181-324, like sgm_uniform.cu).
//
// Each of the eight paths of the two passes (four a pass) is a plain recurrence along lines of the image: path 0 along
// rows, path 2 along columns, paths 1 and 3 along the diagonals. Taken one path at a time, every line is independent: no
// block or warp ever waits for another one. A line is a sequence of pixels a fixed number of pixel indices apart (1, W + 1,
// W or W - 1 for paths 0 to 3): a diagonal that leaves the image at one side goes on at the other side as a new line, so
// that the lines of a path are equally long (to one step) and their addresses linear. On the fast path no sum saturates,
// so the aggregate is the sum of the eight paths in any order.
//
// A lane holds K = 8 planes p0..p7 of its line as u16 pairs (p0, p4), (p1, p5), (p2, p6), (p3, p7) (or K = 4, below): the planes before and
// after a pair's are the neighbouring registers', and only the two at the ends take a byte permute. The aggregates keep
// this order within every K planes until the last read, which puts them in order where they are kept. A step is 47
// cycles of a scheduler (44.3 without its loads; 53.7 with pairs of adjacent planes, 62 with the DPX min/add forms): the
// 16-bit minima and permutes bound it, so the adds are multiply-adds by a kernel-argument one, which issue elsewhere. A
// line takes GL = 4, 8, 16 or 32 lanes (planes / K, rounded
// up to a power of two), so a warp carries 32 / GL neighbouring lines. Two variants, chosen by size (small_form):
//   * small layers: the four paths of a pass in one launch, each adding its L into the aggregates by reductions in L2 (four
//     u16 sums in a 64-bit add, none of which can carry). A pass is as long as one line: latency is what such a layer costs.
//   * large layers, path by path: ckpt_lines walks the lines forward and keeps the path's state every kSeg pixels;
//     pair_lines walks them back in segments of kSeg pixels: it makes the forward L of the segment again from the kept
//     state, adds it in shared memory to the aggregates staged there, then runs the backward recurrence of the other
//     pass over the segment. Forward and backward so share one read and one write of the aggregates: per plane and
//     pixel 22 bytes a layer instead of 36 for eight separate read-modify-write walks, for half as much arithmetic again.
//     The pair walk of a path (bound by HBM) shares its launch with the forward walk of the next one (bound by issue).
//
// The reference's revisits of the last column (revisit_schedule.h): the column's own path-2 chain, with the revisits that
// feed it, runs in one warp of its own beside the other lines; paths 0 and 1 of the revisits read only states of the column
// beside it, kept as the lines pass, and run as independent warps. All of them add into the aggregates by reductions.
#include <algorithm>
#include <cstring>
#include <vector>

#include "common.cuh"
#include "internal.h"
#include "revisit_schedule.h"
#include "lines.cuh"

namespace lux {

namespace {

constexpr int kState = 256;    // u16 of a kept column or edge state (the most planes this form takes)

struct LineArgs {
  int W, H, n, T;
  const uint8_t* raw;
  uint16_t* agg;
  float* depth;
  const float* planes;
  const uchar4* guidance;
  uint32_t p1x2;
  uint32_t one;          // 1: a multiplier the compiler cannot fold
  float p2base;
  float gw[4];
  const uint2* p2t;      // [H][W] P2 of pass +1's paths 0..3 at each pixel; pass -1 crosses the same edges the other way
  uint16_t* ckpt[2];     // [segments][lines][n] forward states, even and odd paths
  uint16_t* ckpt_min[2]; // [segments][lines]
  uint16_t* col_sums;    // [2][H][n] the forward path-2 chains of columns W-1 and 0 (large form)
  uint16_t* edge;        // [3][W][kState] pass +1's states of paths 1..3 at row y_b, read by pass -1's first row
  uint16_t* edge_min;    // [3][W]
  int y_b;
  uint16_t* cs[2];       // per pass [H][2][kState]: N(c-1).p0, N(c-1).p1 (rows of the pass)
  uint16_t* cs_min[2];   // per pass [H][2]
  const int* sched[2];   // per pass: src0, src1, extra (H each), then the revisit rows
  int n_rev[2];
  int keep_agg;
};

template <int K>
LUX_DEV void set_init(Planes<K>& v, uint32_t& md) {
#pragma unroll
  for (int i = 0; i < K / 2; i++) v.r[i] = kInit2;
  md = kInit2;
}
// Planes 0..K-1 one after the other, as the aggregates are kept.
template <int K>
LUX_DEV Planes<K> in_order(const Planes<K>& v) {
  Planes<K> o;
#pragma unroll
  for (int i = 0; i < K / 2; i++) {
    constexpr int N = K / 2;
    const int j = 2 * i % N;  // (pairs of planes 2i, 2i + 1: in the low halves of two registers, then in the high ones)
    o.r[i] = __byte_perm(v.r[j], v.r[j + 1 < N ? j + 1 : j], i < N / 2 ? 0x5410 : 0x7632);
  }
  return o;
}
// A lane's planes in global memory, 2K bytes.
template <int K>
LUX_DEV Planes<K> load_planes(const uint16_t* p) {
  Planes<K> v;
  if constexpr (K == 8) v = as_l4(__ldcg(reinterpret_cast<const uint4*>(p)));
  else {
    const uint2 t = __ldcg(reinterpret_cast<const uint2*>(p));
    v.r[0] = t.x;
    v.r[1] = t.y;
  }
  return v;
}
template <int K>
LUX_DEV void store_planes(uint16_t* p, const Planes<K>& v) {
  if constexpr (K == 8) __stcg(reinterpret_cast<uint4*>(p), as_uint4(v));
  else __stcg(reinterpret_cast<uint2*>(p), make_uint2(v.r[0], v.r[1]));
}

// Adds a lane's u16 sums in L2. No u16 of the aggregates can carry into the next one (every path's L is below 2000).
template <int K>
LUX_DEV void red_add(uint16_t* p, const Planes<K>& v) {  // nothing in the kernel reads the sums
#pragma unroll
  for (int i = 0; i < K / 2; i += 2)
    asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" ::"l"(p + 2 * i), "l"(v.r[i] | ((unsigned long long)v.r[i + 1] << 32)));
}

// A kept state (kState u16 apart): lane gl of the line holds planes K·gl to K·gl + K - 1.
template <int K>
LUX_DEV void put_state(uint16_t* base, uint16_t* mins, size_t i, const Planes<K>& L, uint32_t md, int gl, bool in) {
  if (in) store_planes<K>(base + i * kState + gl * K, L);
  if (gl == 0) __stcg(mins + i, (unsigned short)(md & 0xffffu));
}
template <int K>
LUX_DEV void get_state(const uint16_t* base, const uint16_t* mins, size_t i, Planes<K>& L, uint32_t& md, int gl, bool in) {
  set_init(L, md);
  if (in) L = load_planes<K>(base + i * kState + gl * K);
  md = dup16(__ldcg(mins + i));
}

LUX_DEV float4 guide_at(const LineArgs& a, int x, int y) {
  const uchar4 g = __ldg(a.guidance + (size_t)y * a.W + x);
  return make_float4(g.x, g.y, g.z, g.w);
}
LUX_DEV uint32_t p2_between(const LineArgs& a, float4 g, float4 m) {
  const float gg[4] = {g.x, g.y, g.z, g.w}, mm[4] = {m.x, m.y, m.z, m.w};
  return (uint32_t)sgm_p2(gg, mm, a.gw, a.p2base);
}
LUX_DEV uint32_t p2_entry(const LineArgs& a, int pix, int p) { return __ldg(reinterpret_cast<const uint16_t*>(a.p2t + pix) + p); }

// What pass -1 reads above its first row for path p (1..3) at column x: pass +1's state of row y_b at x + dx.
template <int K>
LUX_DEV void edge_start(const LineArgs& a, int p, int x, Planes<K>& L, uint32_t& md, uint32_t& P2, int gl, bool in) {
  const int xe = x + (p == 1 ? 1 : p == 3 ? -1 : 0);
  set_init(L, md);
  P2 = 0;
  if (a.y_b < 0 || xe < 0 || xe >= a.W) return;
  get_state(a.edge, a.edge_min, (size_t)(p - 1) * a.W + xe, L, md, gl, in);
  P2 = p2_between(a, guide_at(a, x, a.H - 1), guide_at(a, xe, a.y_b));
}

// A column's path-2 chain of one pass by a whole warp, its L added by reductions to sums (image row r at r·stride·n:
// the column's aggregates, or a buffer of its own). SPECIAL: the pass's
// last column (x = W-1 of pass +1, x = 0 of pass -1) with the reference's revisits (revisit_schedule.h). In every T-row
// band of nr rows it visits rows 0..v-1 (v = min(R, nr), R = T - (W-1) mod T), then revisits rows 0..v-1, then visits the
// rest, each reading what the step before left: one chain, except that a band's first revisit reads the newest state of
// the line-buffer half it looks into, which is the last visit's for even v and the one before it for odd v (for v = 1 in
// the first band: the pass's boundary). A revisit also adds its path 3, which restarts from the margin and so equals the
// raw cost.
template <int K, bool BWD, bool SPECIAL>
LUX_DEV void column_chain(const LineArgs& a, int x, int lane, typename RawOf<K>::type* ring, uint16_t* sums, int stride) {
  const int W = a.W, H = a.H, n = a.n, T = a.T;
  const bool in = lane * K < n, first = lane == 0, last = lane * K + K == n;
  const int R = SPECIAL ? T - (W - 1) % T : 0;
  const int full = T + R;  // steps of a whole band
  const int tail = H % T;  // rows of a partial last band
  const int steps = SPECIAL ? (H / T) * full + (tail ? tail + min(R, tail) : 0) : H;
  // step s of the chain: its row of the pass; rev: a revisit; start: a band's first revisit
  auto row_of = [&](int s, bool& rev, bool& start) {
    rev = start = false;
    if (!SPECIAL) return s;
    const int j = s / full, o = s - j * full, base = j * T, v = min(R, min(T, H - base));
    rev = o >= v && o < 2 * v;
    start = o == v;
    return o < v ? base + o : base + o - v;
  };
  auto pix = [&](int t) { return (BWD ? H - 1 - t : t) * W + x; };
  // lane i (mod 8) holds step i of a batch: its row and kind, and the P2 to the row above it in the pass (the table's
  // entry of the lower image row)
  auto load_rows = [&](int b) {
    const int s = b * kBatch + (lane & (kBatch - 1));
    bool rev, start;
    const int t = row_of(min(s, steps - 1), rev, start);
    return t | (rev ? 1 << 29 : 0) | (start ? 1 << 30 : 0);
  };
  auto load_p2 = [&](int rv) {
    const int t = rv & 0x1fffffff;
    return t > 0 ? p2_entry(a, BWD ? pix(t - 1) : pix(t), 2) : 0u;
  };
  // A batch's costs by eight bytes a lane, rows one after the other (a lone warp waits for its instructions more than for
  // anything else: 92 batches of 738 steps at 877 instructions took 146 us).
  using Raw = typename RawOf<K>::type;
  RawRing<K> rr(ring + lane, in);
  const int oct = n >> 3, per_oct = (65536 + oct - 1) / oct;
  auto stage = [&](int b, int rv) {
    for (int c0 = 0; c0 < kBatch * oct; c0 += 32) {
      const int c = c0 + lane, i = (c * per_oct) >> 16, part = c - i * oct;
      const int t = __shfl_sync(0xffffffffu, rv, i & (kBatch - 1)) & 0x1fffffff;
      if (i < kBatch)
        cp_async8(reinterpret_cast<char*>(ring + ((b & 1) * kBatch + i) * 32) + part * 8, a.raw + (size_t)pix(t) * n + part * 8);
    }
    cp_async_commit();
  };
  Planes<K> L, Lp;  // the state, and the state one step before
  uint32_t md, mp, P2start = 0;
  set_init(L, md);
  if (BWD) edge_start(a, 2, x, L, md, P2start, lane, in);
  Lp = L;
  mp = md;
  int rv = load_rows(0), rvn = load_rows(1);
  uint32_t pv = load_p2(rv), pvn = load_p2(rvn);
  stage(0, rv);
  stage(1, rvn);
  const int nb = (steps + kBatch - 1) / kBatch;
  for (int b = 0; b < nb; b++) {
    cp_async_wait<1>();
    __syncwarp();  // (a lane's costs were copied by others)
    const int len = min(kBatch, steps - b * kBatch);
    Raw rb[kBatch];
#pragma unroll
    for (int i = 0; i < kBatch; i++) rb[i] = rr.get(b, i);
    const uint32_t pd = dup16(pv);
    // a whole batch with no band's first revisit, no state to keep and not the pass's start
    const bool plain = b > 0 && len == kBatch &&
                       !__any_sync(0xffffffffu, (rv & (1 << 30)) || (!BWD && (rv & 0x1fffffff) == a.y_b));
    if (plain) {  // its rows follow one another
      uint32_t p2[kBatch];
#pragma unroll
      for (int i = 0; i < kBatch; i++) p2[i] = __shfl_sync(0xffffffffu, pd, i);
      const uint32_t revs = SPECIAL ? __ballot_sync(0xffffffffu, rv & (1 << 29)) : 0u;
      const int t0 = __shfl_sync(0xffffffffu, rv, 0) & 0x1fffffff;
      uint16_t* ap = sums + (size_t)(BWD ? H - 1 - t0 : t0) * stride * n + lane * K;
      const long long ds = (long long)(BWD ? -stride : stride) * n;
#pragma unroll
      for (int i = 0; i < kBatch; i++, ap += ds) {
        Planes<K> raw2;
        unpack(raw2, rb[i]);
        Lp = L;
        mp = md;
        line_step<32>(L, md, raw2, p2[i], a, first, last);
        const uint32_t twice = (revs >> i) & 1u;
        Planes<K> s;
#pragma unroll
        for (int k = 0; k < K / 2; k++) s.r[k] = raw2.r[k] * twice + L.r[k];
        if (in) red_add(ap, s);
      }
    } else {
#pragma unroll 1
      for (int i = 0; i < len; i++) {
        const int ev = __shfl_sync(0xffffffffu, rv, i), t = ev & 0x1fffffff;
        uint32_t p2 = __shfl_sync(0xffffffffu, pv, i);
        if (b == 0 && i == 0) p2 = P2start;
        if (SPECIAL && (ev & (1 << 30))) {
          const int v = min(R, min(T, H - t)), src = (v & 1) ? t + v - 2 : t + v - 1;
          const float4 g = guide_at(a, x, BWD ? H - 1 - t : t);
          if (v & 1) {
            L = Lp;
            md = mp;
          }
          if (src >= 0) {
            p2 = p2_between(a, g, guide_at(a, x, BWD ? H - 1 - src : src));
          } else {
            set_init(L, md);
            p2 = 0;
            if (BWD) edge_start(a, 2, x, L, md, p2, lane, in);
          }
        }
        Planes<K> raw2;
        unpack(raw2, rr.get(b, i));
        Lp = L;
        mp = md;
        line_step<32>(L, md, raw2, dup16(p2), a, first, last);
        if (in) {
          Planes<K> s = L;
          if (SPECIAL && (ev & (1 << 29))) {
#pragma unroll
            for (int k = 0; k < K / 2; k++) s.r[k] += raw2.r[k];
          }
          red_add(sums + (size_t)(BWD ? H - 1 - t : t) * stride * n + lane * K, s);
        }
        if (!BWD && t == a.y_b) put_state(a.edge, a.edge_min, (size_t)1 * W + x, L, md, lane, in);  // the last writer counts
      }
    }
    const int rv2 = load_rows(b + 2);
    __syncwarp();  // every lane has read the batch's costs before they are replaced
    if (b + 2 < nb) stage(b + 2, rv2);
    else cp_async_commit();
    rv = rvn;
    pv = pvn;
    rvn = rv2;
    pvn = load_p2(rv2);
  }
  cp_async_wait<0>();
}

// Paths 0 and 1 of pass PASS's revisits R(c, y), a warp each: their sources are states of column c-1, pass +1's final row,
// or never-written slots.
template <int K, bool BWD>
__global__ void __launch_bounds__(128) k_lines_revisit(const LineArgs a) {
  const int lane = threadIdx.x & 31, k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (k >= a.n_rev[BWD ? 1 : 0]) return;
  const int W = a.W, H = a.H, n = a.n;
  const bool in = lane * K < n, first = lane == 0, last = lane * K + K == n;
  const int* sch = a.sched[BWD ? 1 : 0];
  const int y = sch[3 * H + k];
  const int xc = BWD ? 0 : W - 1, xn = BWD ? 1 : W - 2;  // columns c and c-1 of the pass
  auto row = [&](int t) { return BWD ? H - 1 - t : t; };
  const float4 g = guide_at(a, xc, row(y));
  const size_t pi = (size_t)row(y) * W + xc;
  Planes<K> raw2, sum{};
  using Raw = typename RawOf<K>::type;
  unpack(raw2, in ? __ldg(reinterpret_cast<const Raw*>(a.raw + pi * n) + lane) : RawOf<K>::past());
#pragma unroll
  for (int p = 0; p < 2; p++) {
    const int e = sch[p * H + y], kind = src_kind(e);
    Planes<K> L;
    uint32_t md, p2 = 0;
    set_init(L, md);
    if (kind == kSrcEdge) {
      if (a.y_b >= 0) {
        get_state(a.edge, a.edge_min, xn, L, md, lane, in);
        p2 = p2_between(a, g, guide_at(a, xn, a.y_b));
      }
    } else if (kind != kSrcInit) {
      get_state(a.cs[BWD ? 1 : 0], a.cs_min[BWD ? 1 : 0], (size_t)src_row(e) * 2 + (kind - kSrcCs), L, md, lane, in);
      p2 = p2_between(a, g, guide_at(a, xn, row(src_row(e))));
    }
    line_step<32>(L, md, raw2, dup16(p2), a, first, last);
#pragma unroll
    for (int i = 0; i < K / 2; i++) sum.r[i] += L.r[i];
    // R(y_b) is what pass -1 will read at the last column
    if (!BWD && p == 1 && (sch[2 * H + y] & 1)) put_state(a.edge, a.edge_min, xc, L, md, lane, in);
  }
  if (in) red_add(a.agg + pi * n + lane * K, sum);
}

// Small layers: the four paths of a pass, one launch. Warp 0 takes the special column's path 2, the others 32 / GL lines.
// Latency-bound: a layer this small has one to sixteen warps an SM, and a pass lasts as long as its longest chain.
template <int GL, int K, bool BWD>
__global__ void __launch_bounds__(64) k_lines_pass(const LineArgs a) {
  constexpr int LPW = 32 / GL;
  using Raw = typename RawOf<K>::type;
  __shared__ Raw s_ring[2][2 * kBatch * 32];
  const int W = a.W, H = a.H, n = a.n;
  const int lane = threadIdx.x & 31, gl = lane & (GL - 1), grp = lane / GL;
  Raw* ring = s_ring[threadIdx.x >> 5];
  int wi = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) - 1;
  const int xc = BWD ? 0 : W - 1;  // the pass's last column
  if (wi < 0) {
    column_chain<K, BWD, true>(a, xc, lane, ring, a.agg + (size_t)xc * n, W);
    return;
  }
  int p = 1;
  for (; p < 4; p++) {  // the warps of paths 1, 2, 3, then 0
    const int nw = (line_count(a, p) + LPW - 1) / LPW;
    if (wi < nw) break;
    wi -= nw;
  }
  p &= 3;
  const int NL = line_count(a, p);
  if (wi * LPW >= NL) return;
  const int line0 = wi * LPW + grp, line = min(line0, NL - 1);
  const bool valid = line0 < NL && !(p == 2 && line0 == xc);
  const bool inl = gl * K < n, in = valid && inl, first = gl == 0, last = gl * K + K == n;
  const int NS = line_len(a, p, line);
  Walk w = walk_at(a, p, line_first(a, p, line) + (BWD ? (NS - 1) * line_step_of(p, W) : 0), BWD ? -1 : 1), ws = w;
  RawRing<K> rr(ring + lane, in);
  Planes<K> L;
  uint32_t md, p2prev = 0;
  set_init(L, md);
  if (BWD && p > 0 && w.pi >= W * (H - 1)) edge_start(a, p, w.pi - W * (H - 1), L, md, p2prev, gl, inl);
  p2prev = dup16(p2prev);
  const int steps = __reduce_max_sync(0xffffffffu, NS), nb = (steps + kBatch - 1) / kBatch;
  // P2 of a batch's steps: four of them a lane for GL = 4, one for lane i (mod 8) else
  auto load_p2 = [&](int b, uint32_t (&v)[2]) {
#pragma unroll
    for (int k = 0; k < (GL == 4 ? 2 : 1); k++) {
      const int i = GL == 4 ? gl + 4 * k : gl & (kBatch - 1);
      v[k] = b * kBatch + i < NS ? p2_entry(a, ws.pi + ws.step * i, p) : 0u;
    }
  };
  uint32_t pv[2] = {0, 0}, pvn[2] = {0, 0};
  load_p2(0, pv);
  pv[0] = dup16(pv[0]);
  pv[1] = dup16(pv[1]);
  stage_batch(rr, 0, a.raw, a.n, ws, NS, gl, in);
  ws.advance();
  load_p2(1, pvn);
  stage_batch(rr, 1, a.raw, a.n, ws, NS - kBatch, gl, in);
  ws.advance();
  for (int b = 0; b < nb; b++) {
    cp_async_wait<1>();
    const int t0 = b * kBatch;
    auto p2_at = [&](int i) {
      return GL == 4 ? __shfl_sync(0xffffffffu, pv[i >> 2], i & 3, GL) : __shfl_sync(0xffffffffu, pv[0], i, GL);
    };
    // a whole batch that keeps no state and stays clear of the sides (a new line, column c-1) and of row y_b
    bool odd = t0 + kBatch > NS;
    if (w.dx != 0) odd |= w.dx > 0 ? w.x == 0 || w.x + kBatch > W - 2 : w.x == W - 1 || w.x - kBatch < 2;
    if (p == 0) odd |= t0 + kBatch > W - 2;
    if (!BWD && p > 0) odd |= a.y_b >= 0 && w.pi + w.step * (kBatch - 1) >= a.y_b * W;
    if (!__any_sync(0xffffffffu, odd)) {
      Raw rb[kBatch];
#pragma unroll
      for (int i = 0; i < kBatch; i++) rb[i] = rr.get(b, i);
      uint32_t p2[kBatch];  // (a shuffle between the steps would be waited for)
#pragma unroll
      for (int i = 0; i < kBatch; i++) p2[i] = p2_at(i);
      uint16_t* ap = a.agg + (size_t)w.pi * n + gl * K;
      const long long ds = (long long)w.step * n;
#pragma unroll
      for (int i = 0; i < kBatch; i++, ap += ds) {
        Planes<K> raw2;
        unpack(raw2, rb[i]);
        line_step<GL>(L, md, raw2, BWD ? p2prev : p2[i], a, first, last);
        p2prev = p2[i];
        if (in) red_add(ap, L);
      }
    } else {
      int x = w.x, pi = w.pi;
#pragma unroll
      for (int i = 0; i < kBatch; i++) {
        const bool live = t0 + i < NS;
        // a new line: the pixel at the side the diagonal enters by (but pass -1's last row starts from the edge state)
        if (w.dx != 0 && t0 + i > 0 && x == (w.dx > 0 ? 0 : W - 1)) set_init(L, md);
        Planes<K> raw2;
        unpack(raw2, rr.get(b, i));
        const uint32_t p2 = p2_at(i);
        line_step<GL>(L, md, raw2, BWD ? p2prev : p2, a, first, last);
        p2prev = p2;
        if (in && live) red_add(a.agg + (size_t)pi * n + gl * K, L);
        const int y = p == 0 ? line : p == 2 ? (BWD ? H - 1 - t0 - i : t0 + i) : pi / W;
        if (p < 2) {  // N(c-1): paths 0 and 1 are revisit sources
          const bool at = pi - y * W == (BWD ? 1 : W - 2);
          if (valid && live && at) put_state(a.cs[BWD ? 1 : 0], a.cs_min[BWD ? 1 : 0], (size_t)(BWD ? H - 1 - y : y) * 2 + p, L, md, gl, in);
        }
        if (!BWD && p > 0 && y == a.y_b && valid && live) put_state(a.edge, a.edge_min, (size_t)(p - 1) * W + (pi - y * W), L, md, gl, in);
        pi += w.step;
        x += w.dx;
        if ((unsigned)x >= (unsigned)W) x -= w.dx * W;
      }
    }
    w.advance();
    pv[0] = dup16(pvn[0]);  // the duplication waits for the load: only once the next batch needs it
    pv[1] = dup16(pvn[1]);
    load_p2(b + 2, pvn);
    stage_batch(rr, b + 2, a.raw, a.n, ws, NS - (b + 2) * kBatch, gl, in);
    ws.advance();
  }
  cp_async_wait<0>();
}

template <int GL, int K>
__global__ void __launch_bounds__(256) k_lines_wta(const LineArgs a) {
  constexpr int LPW = 32 / GL;
  const int lane = threadIdx.x & 31, gl = lane & (GL - 1), grp = lane / GL;
  const int npx = a.W * a.H, nwarps = (gridDim.x * blockDim.x) >> 5;
  for (int p0 = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * LPW; p0 < npx; p0 += nwarps * LPW) {
    const int pi = p0 + grp;
    const bool in = pi < npx && gl * K < a.n;
    Planes<K> s{};
    if (in) s = load_planes<K>(a.agg + (size_t)pi * a.n + gl * K);
    const int arg = wta_line<GL>(s, gl, lane, in);
    if (in && gl == 0) a.depth[pi] = __ldg(a.planes + arg);
    if (a.keep_agg && in) store_planes<K>(a.agg + (size_t)pi * a.n + gl * K, in_order(s));
  }
}

// Large layers, forward walk of one path by a warp: its state at the end of every kSeg pixels, and the states that revisits
// and pass -1 read. Bound by issue (55 instructions a step at GL = 32) and, with few lines, by the step's latency.
template <int GL, int P>
LUX_DEV void ckpt_lines(const LineArgs& a, int wi, uint2* ring, uint16_t* ckpt, uint16_t* ckpt_min) {
  constexpr int LPW = 32 / GL;
  static_assert(kBatch == kSeg, "one state a batch");
  const int W = a.W, n = a.n;
  const int lane = threadIdx.x & 31, gl = lane & (GL - 1), grp = lane / GL;
  const int NL = line_count(a, P);
  if (wi * LPW >= NL) return;
  const int line0 = wi * LPW + grp, line = min(line0, NL - 1);
  const bool valid = line0 < NL;
  const bool in = valid && gl * 8 < n, first = gl == 0, last = gl * 8 + 8 == n;
  const int NS = line_len(a, P, line);
  Walk w = walk_at(a, P, line_first(a, P, line), 1), ws = w;
  RawRing<8> rr(ring + lane, in);
  L4 L;
  uint32_t md;
  set_init(L, md);
  const int steps = __reduce_max_sync(0xffffffffu, NS), nb = (steps + kBatch - 1) / kBatch;
  auto load_p2 = [&](int b) {
    const int i = gl & (kBatch - 1);
    return b * kBatch + i < NS ? p2_entry(a, ws.pi + ws.step * i, P) : 0u;
  };
  uint32_t pv = dup16(load_p2(0)), pvn;
  stage_batch(rr, 0, a.raw, a.n, ws, NS, gl, in);
  ws.advance();
  pvn = load_p2(1);
  stage_batch(rr, 1, a.raw, a.n, ws, NS - kBatch, gl, in);
  ws.advance();
  for (int b = 0; b < nb; b++) {
    cp_async_wait<1>();
    const int t0 = b * kBatch;
    bool odd = t0 + kBatch > NS;
    if (P == 1) odd |= w.x == 0 || w.x + kBatch > W - 2;
    if (P == 3) odd |= w.x == W - 1 || w.x < kBatch;
    if (P == 0) odd |= t0 + kBatch > W - 2;
    if (P > 0) odd |= a.y_b >= 0 && w.pi + w.step * (kBatch - 1) >= a.y_b * W;
    if (!__any_sync(0xffffffffu, odd)) {
      uint2 rb[kBatch];
#pragma unroll
      for (int i = 0; i < kBatch; i++) rb[i] = rr.get(b, i);
#pragma unroll
      for (int i = 0; i < kBatch; i++) {
        L4 raw2;
        unpack(raw2, rb[i]);
        line_step<GL>(L, md, raw2, __shfl_sync(0xffffffffu, pv, i, GL), a, first, last);
      }
    } else {
      int x = w.x, pi = w.pi;
#pragma unroll 1
      for (int i = 0; i < kBatch; i++) {
        const bool live = valid && t0 + i < NS;
        if ((P == 1 && x == 0) || (P == 3 && x == W - 1)) set_init(L, md);
        L4 raw2;
        unpack(raw2, rr.get(b, i));
        line_step<GL>(L, md, raw2, __shfl_sync(0xffffffffu, pv, i, GL), a, first, last);
        const int y = P == 0 ? line : P == 2 ? t0 + i : pi / W;
        if (P < 2 && live && pi - y * W == W - 2) put_state(a.cs[0], a.cs_min[0], (size_t)y * 2 + P, L, md, gl, in);
        // (the edge states of path 2's columns 0 and W-1 are their chains')
        if (P > 0 && live && y == a.y_b && !(P == 2 && (line == 0 || line == W - 1)))
          put_state(a.edge, a.edge_min, (size_t)(P - 1) * W + (pi - y * W), L, md, gl, in);
        pi += w.step;
        x += w.dx;
        if ((unsigned)x >= (unsigned)W) x -= w.dx * W;
      }
    }
    if ((b + 1) * kSeg < NS) {
      const size_t ci = (size_t)b * NL + line;
      if (in) __stcs(reinterpret_cast<uint4*>(ckpt + ci * n) + gl, as_uint4(L));
      if (valid && gl == 0) ckpt_min[ci] = (uint16_t)(md & 0xffffu);
    }
    w.advance();
    pv = dup16(pvn);  // the duplication waits for the load: only once the next batch needs it
    pvn = load_p2(b + 2);
    stage_batch(rr, b + 2, a.raw, a.n, ws, NS - (b + 2) * kBatch, gl, in);
    ws.advance();
  }
  cp_async_wait<0>();
}

// Large layers, backward walk of one path by a warp with its forward states made again segment by segment. MODE 0 stores the
// aggregates (the first path of the layer), 1 adds to them, 2 reads them, takes the winner-take-all and stores them only
// when they are kept. Per lane and pixel of a segment: 16 bytes of sums and 8 of raw costs in shared memory, refilled by
// cp.async for the next segment as soon as the backward walk is through with a pixel. Path 2 leaves columns 0 and W-1 to
// their own chains. Bound by HBM (5.6 TB/s for path 1 of 4160x3120 D=256; at 2080x1560 4.5, with issue at 57 %).
template <int GL, int P, int MODE>
LUX_DEV void pair_lines(const LineArgs& a, int wi, uint4* sum, uint2* rawp, const uint16_t* ckpt, const uint16_t* ckpt_min) {
  constexpr int LPW = 32 / GL;
  static_assert(GL >= kSeg, "a lane per pixel of a segment loads its P2");
  const int W = a.W, H = a.H, n = a.n;
  const int lane = threadIdx.x & 31, gl = lane & (GL - 1), grp = lane / GL;
  const int NL = line_count(a, P);
  if (wi * LPW >= NL) return;
  const int line0 = wi * LPW + grp, line = min(line0, NL - 1);
  const bool valid = line0 < NL && !(P == 2 && (line0 == 0 || line0 == W - 1));
  const bool in = valid && gl * 8 < n, first = gl == 0, last = gl * 8 + 8 == n;
  const int NS = line_len(a, P, line), step = line_step_of(P, W);
  const int steps = __reduce_max_sync(0xffffffffu, NS), nseg = (steps + kSeg - 1) / kSeg;
  constexpr int dx = P == 1 ? 1 : P == 3 ? -1 : 0;
  sum += lane;
  rawp += lane;
  if (!in)
    for (int i = 0; i < kSeg; i++) rawp[i * 32] = kPastRaw;
  int pi0 = line_first(a, P, line) + (nseg - 1) * kSeg * step, x0 = dx != 0 ? pi0 % W : 0;  // of the segment in hand
  auto stage = [&](int i, int pi) {
    if (MODE != 0) cp_async16(sum + i * 32, reinterpret_cast<const uint4*>(a.agg + (size_t)pi * n) + gl);
    cp_async8(rawp + i * 32, reinterpret_cast<const uint2*>(a.raw + (size_t)pi * n) + gl);
  };
  for (int i = 0; i < kSeg; i++)
    if (in && (nseg - 1) * kSeg + i < NS) stage(i, pi0 + step * i);
  cp_async_commit();
  auto load_ckpt = [&](int seg, L4& L, uint32_t& mn) {  // the forward state before segment seg, its minimum not yet doubled
    set_init(L, mn);
    if (seg > 0 && seg * kSeg < NS) {
      const size_t ci = (size_t)(seg - 1) * NL + line;
      if (in) L = as_l4(__ldcs(reinterpret_cast<const uint4*>(ckpt + ci * n) + gl));
      mn = __ldcs(ckpt_min + ci);
    }
  };
  auto load_p2 = [&](int seg, int pb) {
    const int i = gl & (kSeg - 1);
    return seg * kSeg + i < NS ? p2_entry(a, pb + step * i, P) : 0u;
  };
  L4 F, B, S;  // the forward and backward states; S, sd, p2start: what the backward walk starts from
  uint32_t fd, bd, sd, p2start = 0;
  load_ckpt(nseg - 1, F, fd);
  fd = dup16(fd);
  uint32_t p2v = dup16(load_p2(nseg - 1, pi0));
  set_init(S, sd);
  const int pl = line_first(a, P, line) + (NS - 1) * step;  // the line's last pixel
  if (P > 0 && pl >= W * (H - 1)) edge_start(a, P, pl - W * (H - 1), S, sd, p2start, gl, gl * 8 < n);
  B = S;
  bd = sd;
  uint32_t p2back = dup16(p2start);  // the P2 of the backward step in hand: the table's entry of the pixel after it
  for (int seg = nseg - 1; seg >= 0; seg--) {
    const int t0 = seg * kSeg;
    cp_async_wait<0>();
    // a whole segment clear of the sides (a new line; column 1, where pass -1's states are kept). Where two lines of a warp end
    // a step apart, one of them is at a side in the segment in which the shorter one ends, whose walk back then starts below.
    bool odd = t0 + kSeg > NS;
    if (P == 1) odd |= x0 <= 1 || x0 + kSeg >= W;
    if (P == 3) odd |= x0 == W - 1 || x0 < kSeg;
    if (P == 0) odd |= t0 <= 1;
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
    // forward, as ckpt_lines walked it
    if (plain) {
#pragma unroll
      for (int i = 0; i < kSeg; i++) {
        L4 raw2;
        unpack(raw2, rawp[i * 32]);
        line_step<GL>(F, fd, raw2, __shfl_sync(0xffffffffu, p2v, i, GL), a, first, last);
        add_fwd(i);
      }
    } else {
      int x = x0;
#pragma unroll 1
      for (int i = 0; i < kSeg; i++) {
        if ((P == 1 && x == 0) || (P == 3 && x == W - 1)) set_init(F, fd);
        L4 raw2;
        unpack(raw2, rawp[i * 32]);
        line_step<GL>(F, fd, raw2, __shfl_sync(0xffffffffu, p2v, i, GL), a, first, last);
        add_fwd(i);
        x += dx;
        if ((unsigned)x >= (unsigned)W) x -= dx * W;
      }
    }
    const int pq = pi0 - step * kSeg;  // the segment before
    L4 Fn;
    uint32_t fdn, p2n = 0;
    load_ckpt(seg - 1, Fn, fdn);
    if (seg > 0) p2n = load_p2(seg - 1, pq);
    int win = 0;  // lane i (mod 8): the winning plane of the segment's pixel i
    auto put = [&](int i, uint16_t* ap, bool live) {  // the pixel's sums: stored, or the winner taken
      L4 s = as_l4(sum[i * 32]);
#pragma unroll
      for (int k = 0; k < 4; k++) s.r[k] += B.r[k];
      if (MODE != 2) {
        if (in && live) __stcs(reinterpret_cast<uint4*>(ap), as_uint4(s));
      } else {
        if (a.keep_agg && in && live) __stcs(reinterpret_cast<uint4*>(ap), as_uint4(in_order(s)));
        const int arg = wta_line<GL>(s, gl, lane, gl * 8 < n);
        if ((gl & (kSeg - 1)) == i) win = arg;
      }
    };
    if (plain) {
      const long long ds = (long long)step * n;
      uint16_t* ap = a.agg + (size_t)(pi0 + step * (kSeg - 1)) * n + gl * 8;
      const uint8_t* rq = a.raw + (size_t)(pq + step * (kSeg - 1)) * n + gl * 8;
#pragma unroll
      for (int i = kSeg - 1; i >= 0; i--, ap -= ds, rq -= ds) {
        L4 raw2;
        unpack(raw2, rawp[i * 32]);
        line_step<GL>(B, bd, raw2, p2back, a, first, last);
        p2back = __shfl_sync(0xffffffffu, p2v, i, GL);
        put(i, ap, true);
        if (in) {
          if (MODE != 0) cp_async16(sum + i * 32, ap - ds * kSeg);
          cp_async8(rawp + i * 32, rq);
        }
      }
    } else {
      int x = x0 + dx * (kSeg - 1), pi = pi0 + step * (kSeg - 1);
      if ((unsigned)x >= (unsigned)W) x -= dx * W;
#pragma unroll 1
      for (int i = kSeg - 1; i >= 0; i--) {
        const bool live = t0 + i < NS;
        if (t0 + i == NS - 1) {  // the line's last pixel: where its backward walk starts
          B = S;
          bd = sd;
          p2back = dup16(p2start);
        } else if ((P == 1 && x == W - 1) || (P == 3 && x == 0)) {
          set_init(B, bd);  // a new line: pass -1 comes in at the side the diagonal left by
        }
        L4 raw2;
        unpack(raw2, rawp[i * 32]);
        line_step<GL>(B, bd, raw2, p2back, a, first, last);
        p2back = __shfl_sync(0xffffffffu, p2v, i, GL);
        put(i, a.agg + (size_t)pi * n + gl * 8, live);
        if (P < 2) {  // N(c-1) of pass -1, column 1
          const int y = P == 0 ? line : pi / W;
          if (valid && live && pi - y * W == 1) put_state(a.cs[1], a.cs_min[1], (size_t)(H - 1 - y) * 2 + P, B, bd, gl, in);
        }
        if (seg > 0 && in && t0 - kSeg + i < NS) stage(i, pq + step * i);
        pi -= step;
        x -= dx;
        if ((unsigned)x >= (unsigned)W) x += dx * W;
      }
    }
    cp_async_commit();
    if (MODE == 2 && valid && gl < kSeg && t0 + gl < NS) a.depth[pi0 + step * gl] = __ldg(a.planes + win);
    F = Fn;
    fd = dup16(fdn);
    p2v = dup16(p2n);
    pi0 = pq;
    x0 -= dx * kSeg;
    if ((unsigned)x0 >= (unsigned)W) x0 += dx * W;
  }
}

// One launch of the large form: the pair walk of path P (its warps first) beside the forward walk of path NEXT, which do
// not depend on each other. P or NEXT = -1: none. The columns 0 and W-1 of path 2 run as chains in the first block: forward,
// beside the forward walk of path 2, into a buffer of their own (the pair walk of path 1 is at the aggregates then);
// backward, beside the pair walk of path 2.
template <int GL, int P, int MODE, int NEXT>
__global__ void __launch_bounds__(64, 16) k_lines_walk(const LineArgs a) {
  constexpr int LPW = 32 / GL;
  constexpr bool kChains = P == 2 || NEXT == 2;
  static_assert(!(P == 2 && NEXT == 2), "one set of chains a launch");
  __shared__ uint4 s_sum[2][kSeg * 32];
  __shared__ uint2 s_raw[2][kSeg * 32];
  const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint2* ring = reinterpret_cast<uint2*>(s_sum[wib]);
  int block = blockIdx.x;
  if (kChains) {
    if (block == 0) {
      const int x = wib == 0 ? a.W - 1 : 0;
      if (NEXT == 2) {
        uint16_t* sums = a.col_sums + (size_t)wib * a.H * a.n;
        if (wib == 0) column_chain<8, false, true>(a, x, lane, ring, sums, 1);
        else column_chain<8, false, false>(a, x, lane, ring, sums, 1);
      } else {
        uint16_t* sums = a.agg + (size_t)x * a.n;
        if (wib == 0) column_chain<8, true, false>(a, x, lane, ring, sums, a.W);
        else column_chain<8, true, true>(a, x, lane, ring, sums, a.W);
      }
      return;
    }
    block--;
  }
  constexpr int PP = P < 0 ? 0 : P, PN = NEXT < 0 ? 0 : NEXT;
  const int pair_blocks = P < 0 ? 0 : ((line_count(a, PP) + LPW - 1) / LPW + 1) / 2;
  if (P >= 0 && block < pair_blocks) {
    pair_lines<GL, PP, MODE>(a, block * 2 + wib, s_sum[wib], s_raw[wib], a.ckpt[PP & 1], a.ckpt_min[PP & 1]);
  } else if (NEXT >= 0) {
    ckpt_lines<GL, PN>(a, (block - pair_blocks) * 2 + wib, ring, a.ckpt[PN & 1], a.ckpt_min[PN & 1]);
  }
}

// Adds the forward chains of columns W-1 and 0 into the aggregates (a thread per eight planes).
__global__ void k_lines_columns(const LineArgs a) {
  const int oct = a.n / 8, i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= 2 * a.H * oct) return;
  const int c = i / (a.H * oct), j = i - c * a.H * oct, y = j / oct;
  const L4 v = as_l4(__ldcg(reinterpret_cast<const uint4*>(a.col_sums) + i));
  red_add(a.agg + ((size_t)y * a.W + (c == 0 ? a.W - 1 : 0)) * a.n + (j - y * oct) * 8, v);
}

struct LinesLayout {
  size_t ckpt[2], ckpt_min[2], col_sums, edge, edge_min, cs, cs_min, sched, p2t, total;
};
// The small form's eight reductions a value cost 8 us a million planes and pixels at any size; the large form moves less
// but walks path after path. Small against large, ms: 2080x1560 D=64 1.6 / 2.7, D=96 2.5 / 2.9, D=128 3.0 / 3.1, 3000x2000 D=64
// 3.3 / 3.5, 4160x3120 D=40 5.1 / 5.5, D=64 6.6 / 5.8, D=128 12.8 / 9.0; past 128 planes, where a lane holds eight in either
// form, 1431x1073 D=200 3.0 / 2.3. With 32 planes or fewer the large form's lines leave lanes idle: 4160x3120 D=32 3.1 / 5.6.
bool small_form(int W, int H, int n) {
  return W < 2 * kSeg || n <= 32 || (size_t)W * H * n < (size_t)(n <= 128 ? 480 : 240) << 20;
}

LinesLayout lines_layout(int W, int H, int n, bool keep_states) {
  auto al = [](size_t v) { return (v + 255) & ~(size_t)255; };
  LinesLayout s;
  size_t o = 0;
  // states: W + 1 lines or fewer of at most H + H / (W - 1) + 1 steps, or H lines of W
  const size_t states = !keep_states ? 0 : std::max((size_t)(W + 1) * ((H + H / (W - 1) + 1) / kSeg + 1), (size_t)H * (W / kSeg + 1));
  for (int k = 0; k < 2; k++) {
    s.ckpt[k] = o; o += al(states * n * 2);
    s.ckpt_min[k] = o; o += al(states * 2);
  }
  s.col_sums = o; o += states ? al((size_t)2 * H * n * 2) : 0;
  s.edge = o; o += al((size_t)3 * W * kState * 2);
  s.edge_min = o; o += al((size_t)3 * W * 2);
  s.cs = o; o += al((size_t)2 * H * 2 * kState * 2);
  s.cs_min = o; o += al((size_t)2 * H * 2 * 2);
  s.sched = o; o += al((size_t)2 * 4 * H * 4);
  s.p2t = o; o += al((size_t)W * H * 8);
  s.total = o;
  return s;
}

template <int GL, int K>
void run_small(const LineArgs& a, cudaStream_t s) {
  constexpr int LPW = 32 / GL;
  auto warps_of = [](int lines) { return (lines + LPW - 1) / LPW; };
  const int blocks = (1 + warps_of(a.W + 1) + warps_of(a.W) + warps_of(a.W - 1) + warps_of(a.H) + 1) / 2;
  cudaMemsetAsync(a.agg, 0, (size_t)a.W * a.H * a.n * 2, s);
  k_lines_pass<GL, K, false><<<blocks, 64, 0, s>>>(a);
  if (a.n_rev[0]) k_lines_revisit<K, false><<<(a.n_rev[0] + 3) / 4, 128, 0, s>>>(a);
  k_lines_pass<GL, K, true><<<blocks, 64, 0, s>>>(a);
  if (a.n_rev[1]) k_lines_revisit<K, true><<<(a.n_rev[1] + 3) / 4, 128, 0, s>>>(a);
  const int wta = (a.W * a.H + 8 * LPW - 1) / (8 * LPW);
  k_lines_wta<GL, K><<<std::min(wta, 148 * 8), 256, 0, s>>>(a);
  count_launches(3 + (a.n_rev[0] > 0) + (a.n_rev[1] > 0));
}

template <int GL, int P, int MODE, int NEXT>
void run_walk(const LineArgs& a, cudaStream_t s) {
  constexpr int LPW = 32 / GL;
  auto blocks_of = [&](int p) {
    const int lines = p < 0 ? 0 : p == 0 ? a.H : p == 1 ? a.W + 1 : p == 2 ? a.W : a.W - 1;
    return ((lines + LPW - 1) / LPW + 1) / 2;
  };
  k_lines_walk<GL, P, MODE, NEXT><<<blocks_of(P) + blocks_of(NEXT) + (P == 2 || NEXT == 2 ? 1 : 0), 64, 0, s>>>(a);
  count_launches(1);
}
template <int GL>
void run_large(const LineArgs& a, cudaStream_t s) {
  cudaMemsetAsync(a.col_sums, 0, (size_t)2 * a.H * a.n * 2, s);
  run_walk<GL, -1, 0, 0>(a, s);
  run_walk<GL, 0, 0, 1>(a, s);
  // pass -1's diagonals from the last column start at what the last revisit left there
  if (a.n_rev[0]) k_lines_revisit<8, false><<<(a.n_rev[0] + 3) / 4, 128, 0, s>>>(a);
  run_walk<GL, 1, 1, 2>(a, s);
  if (a.n_rev[1]) k_lines_revisit<8, true><<<(a.n_rev[1] + 3) / 4, 128, 0, s>>>(a);
  run_walk<GL, 2, 1, 3>(a, s);
  k_lines_columns<<<(2 * a.H * (a.n / 8) + 255) / 256, 256, 0, s>>>(a);
  run_walk<GL, 3, 2, -1>(a, s);
  count_launches(1 + (a.n_rev[0] > 0) + (a.n_rev[1] > 0));
}

}  // namespace

// The layers this form takes, beyond uniform_fast_supported's: at most 256 planes, and rows of a batch's length or more (a
// diagonal wraps at most once in a batch).
bool lines_supported(int W, int n) { return n <= kState && W >= kBatch; }
bool lines_keep_states(int W, int H, int n) { return !small_form(W, H, n); }
size_t lines_scratch_bytes(int W, int H, int n, bool keep_states) { return lines_layout(W, H, n, keep_states).total; }

// k_p2_table lives in sgm_uniform.cu
void launch_p2_table(const UniArgs& a, uint2* p2t, cudaStream_t s);

int run_sgm_lines(const LayerGeom& g, uint16_t p1, float p2scale, const float gw[4], const uint8_t* raw, uint16_t* agg, float* depth,
                  int keep_agg, bool keep_states, void* scratch, size_t scratch_bytes, cudaStream_t s) {
  const int W = g.W, H = g.H, n = g.n_planes, T = g.tile;
  const LinesLayout L = lines_layout(W, H, n, keep_states);
  if (scratch_bytes < L.total) return 9;
  char* base = static_cast<char*>(scratch);
  LineArgs a;
  std::memset(&a, 0, sizeof a);
  std::vector<int> host((size_t)2 * 4 * H, 0);
  RevisitSchedule sch;
  int* dsched = reinterpret_cast<int*>(base + L.sched);
  for (int pass = 0; pass < 2; pass++) {
    build_revisit_schedule(W, H, T, pass == 1, sch);
    if (pass == 0) a.y_b = sch.y_b;
    int* h = host.data() + (size_t)pass * 4 * H;
    const std::vector<int>* cols[3] = {&sch.src0, &sch.src1, &sch.extra};
    for (int k = 0; k < 3; k++) std::memcpy(h + (size_t)k * H, cols[k]->data(), (size_t)H * 4);
    int* rl = h + (size_t)3 * H;
    for (int y = 0; y < H; y++)
      for (int k = 0; k < sch.batch_count[y]; k++) rl[a.n_rev[pass]++] = sch.batch_first[y] + k;
    for (int k = 0; k < sch.end_count; k++) rl[a.n_rev[pass]++] = sch.end_first + k;
    a.sched[pass] = dsched + (size_t)pass * 4 * H;
    a.cs[pass] = reinterpret_cast<uint16_t*>(base + L.cs) + (size_t)pass * H * 2 * kState;
    a.cs_min[pass] = reinterpret_cast<uint16_t*>(base + L.cs_min) + (size_t)pass * H * 2;
  }
  if (cudaMemcpyAsync(dsched, host.data(), host.size() * 4, cudaMemcpyHostToDevice, s) != cudaSuccess) return 10;
  a.W = W; a.H = H; a.n = n; a.T = T;
  a.raw = raw; a.agg = agg; a.depth = depth; a.planes = g.planes; a.guidance = g.guidance;
  a.p1x2 = (uint32_t)p1 * 0x10001u;
  a.one = 1;
  volatile float p1f = (float)p1;
  a.p2base = p1f * p2scale;
  for (int i = 0; i < 4; i++) a.gw[i] = gw[i];
  a.p2t = reinterpret_cast<const uint2*>(base + L.p2t);
  for (int k = 0; k < 2; k++) {
    a.ckpt[k] = reinterpret_cast<uint16_t*>(base + L.ckpt[k]);
    a.ckpt_min[k] = reinterpret_cast<uint16_t*>(base + L.ckpt_min[k]);
  }
  a.col_sums = reinterpret_cast<uint16_t*>(base + L.col_sums);
  a.edge = reinterpret_cast<uint16_t*>(base + L.edge);
  a.edge_min = reinterpret_cast<uint16_t*>(base + L.edge_min);
  a.keep_agg = keep_agg;
  UniArgs u;
  std::memset(&u, 0, sizeof u);
  u.W = W; u.H = H; u.dir = 1; u.guidance = g.guidance; u.p2base = a.p2base; u.y_b = -1;
  for (int i = 0; i < 4; i++) u.gw[i] = gw[i];
  launch_p2_table(u, reinterpret_cast<uint2*>(base + L.p2t), s);
  if (!keep_states) {
    // four planes a lane up to 128: half the instructions a step of eight, for twice the warps (ms, four / eight: 520x390 D=32
    // 0.27 / 0.29, 1431x1073 D=64 0.93 / 0.96, 1600x1200 D=128 1.85 / 2.12, 2080x1560 D=64 1.6 / 1.9, 4160x3120 D=32 3.1 / 4.2)
    if (n <= 16) run_small<4, 4>(a, s);
    else if (n <= 32) run_small<8, 4>(a, s);
    else if (n <= 64) run_small<16, 4>(a, s);
    else if (n <= 128) run_small<32, 4>(a, s);
    else run_small<32, 8>(a, s);
  } else {
    if (n <= 64) run_large<8>(a, s);
    else if (n <= 128) run_large<16>(a, s);
    else run_large<32>(a, s);
  }
  return 0;
}

}  // namespace lux
