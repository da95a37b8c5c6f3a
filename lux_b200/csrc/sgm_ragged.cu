// Aggregation of a ragged layer (every pixel searches its own plane range) by single lines, like sgm_lines.cu's small form:
// every path of a pass is walked along its own independent lines and added into the aggregates by reductions in L2. Also
// uniform layers of more planes than sgm_lines.cu's lanes hold. Bit-exact with the reference's traversal (sgm_emulate.cu)
// where that is a plain recurrence over the pixels' ranges:
//
// The reference keeps a pixel's four path states in a flat line buffer, a block of MaxHi + 1 planes a path; a pixel reads
// its neighbour's block at its own planes -1 .. +1. What lies there is the neighbour's L inside the neighbour's range and
// 2000 outside (a pixel first clears the range stored in its slot before), unless a range reaches past the block's last
// plane: then writes spill into the next block (or slot), and reads past the block see what the next path keeps at its
// first planes. k_ragged_check looks for pixels that touch plane MaxHi or beyond ("high": q + cap > MaxHi, q the start
// less MinLo). Such a pixel, and the pixels that read it, still see plain values when nothing near it touches the first
// planes of a block: no pixel within two rows and columns starts at plane 7 or below (the spill is at most seven planes
// long; two rows up is what the slot held before), and it is not within two pixels of the image's border (the revisits of
// the last column, the first rows' initial state, the rows that pass -1 starts from). Layers where this does not hold, or
// with a pixel of no planes, take the exact replay.
//
// A warp walks a line. The path's state lies in shared memory by plane, twice (a pixel's step reads one copy and writes the
// other); a lane takes an aligned quad of the block's planes, 128 planes a round, and only the rounds a pixel's range
// touches run. Raw costs come through shared memory too, staged by cp.async a batch of pixels ahead; the ranges, offsets
// and P2 of a batch are one 16-byte load a lane, two batches ahead. The aggregates' quads start at the pixel's first plane,
// the lanes' at the block's: the sums are read back from the state at the pixel's own alignment. Bound by issue and, with
// few lines, by the step's latency (about 200 instructions a pixel and path of up to 128 planes). The finest layer of a
// 2080x1560 capture (65 planes a pixel): 3.8 + 3.5 ms for the two passes, 54 ms on the replay.
#include <algorithm>
#include <cstring>
#include <vector>

#include "common.cuh"
#include "internal.h"
#include "revisit_schedule.h"
#include "sgm_paths.cuh"

namespace lux {

namespace {

constexpr int kBatch = 4;       // pixels of a batch
constexpr int kRound = 128;     // planes of a round: 32 lanes of four
constexpr int kMaxRounds = 7;
constexpr int kLead = 4;        // u16 before plane 0 of a state copy
constexpr int kPad = 8;         // bytes before a pixel's raw costs in its ring slot (a quad's first byte may lie 3 before)

struct RagArgs {
  int W, H, T, y_b;
  const uint4* info;     // per pixel {offset / 8, q | cap << 16, P2 of paths 0 | 1 << 16, 2 | 3 << 16}
  const uint8_t* raw;
  uint16_t* agg;
  const uchar4* guidance;
  uint32_t p1x2, one;    // one = 1: a multiplier the compiler cannot fold (multiply-adds issue beside the minima)
  float p2base;
  float gw[4];
  uint16_t* edge;        // [3][W][state] pass +1's states of paths 1..3 at row y_b
  uint16_t* edge_min;    // [3][W]
  uint16_t* cs[2];       // per pass [H][2][state]: N(c-1).p0, N(c-1).p1 (rows of the pass)
  uint16_t* cs_min[2];   // per pass [H][2]
  const int* sched[2];   // per pass: src0, src1, extra (H each), then the revisit rows
  int n_rev[2];
  int rounds;            // of the layer's planes: a state is rounds · kRound u16
  int ring_bytes;        // a pixel's slot of raw costs in shared memory
};

// A warp's path state: the current copy, with the rounds that may hold anything but 2000, the other copy with its own, and
// the least L in both halves.
struct RState {
  uint16_t *cur, *oth;
  int lo, hi, olo, ohi;
  uint32_t md;
  LUX_DEV void flip() {
    uint16_t* t = cur;
    cur = oth;
    oth = t;
    const int l = lo, h = hi;
    lo = olo;
    hi = ohi;
    olo = l;
    ohi = h;
  }
};
__host__ __device__ constexpr int state_u16(int rounds) { return rounds * kRound + 2 * kLead; }
LUX_DEV void clear_rounds(uint16_t* p, int lo, int hi, int lane) {
#pragma unroll 1
  for (int j = lo; j <= hi; j++) reinterpret_cast<uint2*>(p)[j * 32 + lane] = make_uint2(kInit2, kInit2);
}
LUX_DEV void state_new(RState& s, const RagArgs& a, uint16_t* buf, int lane) {  // both copies never written
  const int n = state_u16(a.rounds);
  for (int i = lane; i < n; i += 32) reinterpret_cast<uint32_t*>(buf)[i] = kInit2;
  s.cur = buf + kLead;
  s.oth = s.cur + n;
  s.lo = s.olo = 1;
  s.hi = s.ohi = 0;
  s.md = kInit2;
  __syncwarp();
}
LUX_DEV void state_init(RState& s, int lane) {
  __syncwarp();  // the copy has been read (ragged_add: a lane's planes lie in other lanes' quads)
  clear_rounds(s.cur, s.lo, s.hi, lane);
  s.lo = 1;
  s.hi = 0;
  s.md = kInit2;
  __syncwarp();
}
LUX_DEV void state_put(const RagArgs& a, uint16_t* base, uint16_t* mins, size_t i, const RState& s, int lane) {
#pragma unroll 1
  for (int j = 0; j < a.rounds; j++)
    __stcg(reinterpret_cast<uint2*>(base + (i * a.rounds + j) * kRound) + lane, reinterpret_cast<const uint2*>(s.cur)[j * 32 + lane]);
  if (lane == 0) __stcg(mins + i, (unsigned short)(s.md & 0xffffu));
}
LUX_DEV void state_get(const RagArgs& a, const uint16_t* base, const uint16_t* mins, size_t i, RState& s, int lane) {
#pragma unroll 1
  for (int j = 0; j < a.rounds; j++)
    reinterpret_cast<uint2*>(s.cur)[j * 32 + lane] = __ldcg(reinterpret_cast<const uint2*>(base + (i * a.rounds + j) * kRound) + lane);
  s.lo = 0;
  s.hi = a.rounds - 1;
  s.md = dup16(__ldcg(mins + i));
  __syncwarp();
}

// A pixel's range: q..q+cap-1 of the block's planes.
struct Range {
  int q, cap;
  LUX_DEV Range(uint32_t qc) : q(qc & 0xffff), cap(qc >> 16) {}
};

// One path step to a pixel of range g (DenseStereoSgm.cs:258-315): reads the current copy, writes the other one (2000
// outside the range) and makes it current. rawp: the pixel's ring slot (plane k of the range at byte kPad + k).
LUX_DEV void ragged_step(RState& s, const Range& g, uint32_t p2, const uint8_t* rawp, const RagArgs& a, int lane) {
  const uint32_t one = a.one, neg = 0u - a.one, md = s.md, p2x = dup16(p2) * one + md;
  const int Q0 = g.q >> 2, Q1 = (g.q + g.cap - 1) >> 2, sh = g.q & 3, j0 = Q0 >> 5, j1 = Q1 >> 5, quads = g.cap >> 2;
  const uint32_t sel = 0x3210u + 0x1111u * (4 - sh);
  // the planes in the range of the first quad (from plane sh on) and of the last one (below sh; all when sh = 0)
  const uint32_t f0 = sh == 0 ? 0xffffffffu : sh == 1 ? 0xffff0000u : 0u, f1 = sh <= 2 ? 0xffffffffu : 0xffff0000u;
  const uint32_t l0 = sh == 0 ? 0xffffffffu : ~f0, l1 = sh == 0 ? 0xffffffffu : ~f1;
  const uint16_t* src = s.cur;
  uint16_t* dst = s.oth;
  if (s.olo < j0 || s.ohi > j1) {  // what the other copy holds outside this range's rounds
    clear_rounds(dst, s.olo, min(s.ohi, j0 - 1), lane);
    clear_rounds(dst, max(s.olo, j1 + 1), s.ohi, lane);
  }
  uint32_t m = kInit2;
  auto round = [&](int j) {
    const int quad = 32 * j + lane;
    const uint2 n = reinterpret_cast<const uint2*>(src)[quad];
    const uint32_t before = *reinterpret_cast<const uint32_t*>(src + 4 * quad - 2), after = *reinterpret_cast<const uint32_t*>(src + 4 * quad + 4);
    const uint32_t* rp = reinterpret_cast<const uint32_t*>(rawp + kPad) + min(max(quad - Q0, 0), quads);
    const uint32_t w = __byte_perm(rp[-1], rp[0], sel);
    const uint32_t A = __byte_perm(before, n.x, 0x5432), B = __byte_perm(n.x, n.y, 0x5432), C = __byte_perm(n.y, after, 0x5432);
    const bool inside = quad > Q0 && quad < Q1;
    const uint32_t m0 = inside ? 0xffffffffu : quad == Q0 ? f0 : quad == Q1 ? l0 : 0u;
    const uint32_t m1 = inside ? 0xffffffffu : quad == Q0 ? f1 : quad == Q1 ? l1 : 0u;
    const uint32_t t0 = vmin2(vmin2(vmin2(A, B) * one + a.p1x2, n.x), p2x) * one + (md * neg + __byte_perm(w, 0, 0x4140));
    const uint32_t t1 = vmin2(vmin2(vmin2(B, C) * one + a.p1x2, n.y), p2x) * one + (md * neg + __byte_perm(w, 0, 0x4342));
    const uint32_t o0 = (t0 & m0) | (kInit2 & ~m0), o1 = (t1 & m1) | (kInit2 & ~m1);
    reinterpret_cast<uint2*>(dst)[quad] = make_uint2(o0, o1);
    m = vmin2(m, vmin2(o0, o1));
  };
  round(j0);
#pragma unroll 1
  for (int j = j0 + 1; j <= j1; j++) round(j);
  m = vmin2(m, __byte_perm(m, 0, 0x1032));
  s.md = __reduce_min_sync(0xffffffffu, m);
  s.flip();
  s.lo = j0;
  s.hi = j1;
  __syncwarp();  // the new copy is every lane's, and the old one read
}

// Adds the pixel's L into its aggregates, and with `twice` its raw costs too (a revisit's path 3).
LUX_DEV void ragged_add(const RState& s, const Range& g, uint16_t* agg, bool twice, const uint8_t* rawp, int lane) {
  const uint32_t* src = reinterpret_cast<const uint32_t*>(s.cur) + (g.q >> 1);
  const uint32_t sel = g.q & 1 ? 0x5432u : 0x3210u;
  auto add = [&](int w) {
    const uint32_t s0 = src[2 * w], s1 = src[2 * w + 1], s2 = src[2 * w + 2];
    uint32_t n0 = __byte_perm(s0, s1, sel), n1 = __byte_perm(s1, s2, sel);
    if (twice) {
      const uint32_t r = reinterpret_cast<const uint32_t*>(rawp + kPad)[w];
      n0 += __byte_perm(r, 0, 0x4140);
      n1 += __byte_perm(r, 0, 0x4342);
    }
    const unsigned long long v = n0 | ((unsigned long long)n1 << 32);
    asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" ::"l"(agg + w * 4), "l"(v));  // nothing in the kernel reads them
  };
  const int quads = g.cap >> 2;
  if (lane < quads) add(lane);
  if (quads > 32)
#pragma unroll 1
    for (int w = lane + 32; w < quads; w += 32) add(w);
}

LUX_DEV uint32_t p2_between(const RagArgs& a, int x, int y, int xn, int yn) {
  const uchar4 g = __ldg(a.guidance + (size_t)y * a.W + x), m = __ldg(a.guidance + (size_t)yn * a.W + xn);
  const float gg[4] = {(float)g.x, (float)g.y, (float)g.z, (float)g.w}, mm[4] = {(float)m.x, (float)m.y, (float)m.z, (float)m.w};
  return (uint32_t)sgm_p2(gg, mm, a.gw, a.p2base);
}

// What pass -1 reads above its first row for path p (1..3) at column x: pass +1's state of row y_b at x + dx.
LUX_DEV void edge_start(const RagArgs& a, int p, int x, RState& s, uint32_t& P2, int lane) {
  const int xe = x + (p == 1 ? 1 : p == 3 ? -1 : 0);
  state_init(s, lane);
  P2 = 0;
  if (a.y_b < 0 || xe < 0 || xe >= a.W) return;
  state_get(a, a.edge, a.edge_min, (size_t)(p - 1) * a.W + xe, s, lane);
  P2 = p2_between(a, x, a.H - 1, xe, a.y_b);
}

// Per batch and lane i (mod kBatch): pixel i's aggregate offset / 8, its range and the P2 of the path in hand.
struct Px {
  uint32_t off8, qc, p2;
};
LUX_DEV Px load_px(const RagArgs& a, int pi, int p, bool live) {
  Px v{0u, 8u << 16, 0u};
  if (live) {
    const uint4 t = __ldg(a.info + pi);
    v.off8 = t.x;
    v.qc = t.y;
    v.p2 = p < 2 ? t.z : t.w;  // both paths of the word: taken apart when used, so that nothing waits here
  }
  return v;
}
LUX_DEV uint8_t* ring_slot(const RagArgs& a, uint8_t* ring, int b, int i) { return ring + ((b & 1) * kBatch + i) * a.ring_bytes; }
LUX_DEV void stage_px(const RagArgs& a, uint8_t* ring, int b, const Px& v, int len, int lane) {
#pragma unroll
  for (int i = 0; i < kBatch; i++) {
    const uint32_t off8 = __shfl_sync(0xffffffffu, v.off8, i);
    const int octs = (int)(__shfl_sync(0xffffffffu, v.qc, i) >> 19);
    if (i < len) {
      uint8_t* d = ring_slot(a, ring, b, i) + kPad + lane * 8;
      const uint8_t* src = a.raw + ((size_t)off8 + lane) * 8;
      if (lane < octs) cp_async8(d, src);
      if (octs > 32)
#pragma unroll 1
        for (int o = 32; o + lane < octs; o += 32) cp_async8(d + o * 8, src + o * 8);
    }
  }
  cp_async_commit();
}

// A column's path-2 chain of one pass with the revisits of the pass's last column, in the order and from the sources that
// sgm_lines.cu's column_chain describes.
template <bool BWD>
LUX_DEV void ragged_chain(const RagArgs& a, int x, int lane, uint8_t* ring, RState& s) {
  const int W = a.W, H = a.H, T = a.T;
  const int K = T - (W - 1) % T, full = T + K, tail = H % T;
  const int steps = (H / T) * full + (tail ? tail + min(K, tail) : 0);
  auto pix = [&](int t) { return (BWD ? H - 1 - t : t) * W + x; };
  auto load_row = [&](int b) {  // lane i (mod kBatch): step i's row of the pass; bit 29: a revisit, bit 30: a band's first one
    const int s = min(b * kBatch + (lane & (kBatch - 1)), steps - 1);
    const int j = s / full, o = s - j * full, base = j * T, v = min(K, min(T, H - base));
    return (o < v ? base + o : base + o - v) | (o >= v && o < 2 * v ? 1 << 29 : 0) | (o == v ? 1 << 30 : 0);
  };
  auto load_p2 = [&](int rv) {  // the P2 to the row above in the pass: the entry of the lower image row
    const int t = rv & 0x1fffffff;
    return t > 0 ? __ldg(&a.info[BWD ? pix(t - 1) : pix(t)].w) : 0u;
  };
  uint32_t P2start = 0, md_before = kInit2;  // the other copy holds the state one step before
  if (BWD) edge_start(a, 2, x, s, P2start, lane);
  int rv0 = load_row(0), rv1 = load_row(1), rv2 = load_row(2);
  Px v0 = load_px(a, pix(rv0 & 0x1fffffff), 2, true), v1 = load_px(a, pix(rv1 & 0x1fffffff), 2, true),
     v2 = load_px(a, pix(rv2 & 0x1fffffff), 2, true);
  uint32_t p0 = load_p2(rv0), p1 = load_p2(rv1), p2 = load_p2(rv2);
  stage_px(a, ring, 0, v0, kBatch, lane);
  stage_px(a, ring, 1, v1, kBatch, lane);
  const int nb = (steps + kBatch - 1) / kBatch;
  for (int b = 0; b < nb; b++) {
    cp_async_wait<1>();
    __syncwarp();
    const int len = min(kBatch, steps - b * kBatch);
#pragma unroll 1
    for (int i = 0; i < len; i++) {
      const int ev = __shfl_sync(0xffffffffu, rv0, i), t = ev & 0x1fffffff;
      uint32_t P2 = __shfl_sync(0xffffffffu, p0, i) & 0xffffu;
      if (b == 0 && i == 0) P2 = P2start;
      if (ev & (1 << 30)) {
        const int v = min(K, min(T, H - t)), src = (v & 1) ? t + v - 2 : t + v - 1;
        if ((v & 1) && src >= 0) {
          __syncwarp();  // the copy that the next step writes has been read
          s.flip();
          s.md = md_before;
        }
        if (src >= 0) {
          P2 = p2_between(a, x, BWD ? H - 1 - t : t, x, BWD ? H - 1 - src : src);
        } else {
          state_init(s, lane);
          P2 = 0;
          if (BWD) edge_start(a, 2, x, s, P2, lane);
        }
      }
      const Range g(__shfl_sync(0xffffffffu, v0.qc, i));
      const uint32_t off8 = __shfl_sync(0xffffffffu, v0.off8, i);
      const uint8_t* rawp = ring_slot(a, ring, b, i);
      md_before = s.md;
      ragged_step(s, g, P2, rawp, a, lane);
      ragged_add(s, g, a.agg + (size_t)off8 * 8, (ev & (1 << 29)) != 0, rawp, lane);
      if (!BWD && t == a.y_b) state_put(a, a.edge, a.edge_min, (size_t)1 * W + x, s, lane);  // the last writer counts
    }
    __syncwarp();  // every lane has read the batch's costs before they are replaced
    rv0 = rv1;
    v0 = v1;
    p0 = p1;
    rv1 = rv2;
    v1 = v2;
    p1 = p2;
    stage_px(a, ring, b + 2, v1, b + 2 < nb ? kBatch : 0, lane);
    rv2 = load_row(b + 3);
    v2 = load_px(a, pix(rv2 & 0x1fffffff), 2, true);
    p2 = load_p2(rv2);
  }
  cp_async_wait<0>();
}

// A pixel's ring slot: a range is at most MaxHi + 7 long; a quad may read a word past it.
constexpr int ring_bytes_of(int max_hi) { return (kPad + max_hi + 8 + 8 + 15) & ~15; }
__host__ __device__ constexpr int warp_smem(int rounds, int ring_bytes) { return 2 * kBatch * ring_bytes + ((2 * state_u16(rounds) * 2 + 15) & ~15); }

// The four paths of a pass, a warp a line; warp 0 takes the special column's path 2.
template <bool BWD>
__global__ void __launch_bounds__(64) k_ragged_pass(const RagArgs a) {
  extern __shared__ __align__(16) uint8_t smem_ragged[];
  const int W = a.W, H = a.H, lane = threadIdx.x & 31;
  uint8_t* ring = smem_ragged + (size_t)(threadIdx.x >> 5) * warp_smem(a.rounds, a.ring_bytes);
  RState s;
  state_new(s, a, reinterpret_cast<uint16_t*>(ring + 2 * kBatch * a.ring_bytes), lane);
  int line = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5) - 1;
  const int xc = BWD ? 0 : W - 1, dir = BWD ? -1 : 1;
  if (line < 0) {
    ragged_chain<BWD>(a, xc, lane, ring, s);
    return;
  }
  // the lines of sgm_lines.cu: W + 1, W, W - 1 and H of them for paths 1, 2, 3 and 0
  int p = 1, lines = W + 1;
  while (p < 4 && line >= lines) {
    line -= lines;
    p++;
    lines--;
  }
  p &= 3;
  if (p == 0 && line >= H) return;
  if (p == 2 && line == xc) return;
  const int step = p == 0 ? 1 : p == 1 ? W + 1 : p == 2 ? W : W - 1;
  const int len = p == 0 ? W : p == 2 ? H : (W * H - line + step - 1) / step;
  const int pi0 = (p == 0 ? line * W : line) + (BWD ? (len - 1) * step : 0);
  const int dx = p < 2 ? dir : p == 3 ? -dir : 0, dy = p == 0 ? 0 : dir, turn = p == 1 ? dir : -dir;  // turn: dy's change at a side
  int y = pi0 / W, x = pi0 - y * W;
  uint32_t p2prev = 0;
  if (BWD && p > 0 && y == H - 1) edge_start(a, p, x, s, p2prev, lane);
  auto load = [&](int b) {
    const int i = b * kBatch + (lane & (kBatch - 1));
    return load_px(a, pi0 + dir * step * i, p, i < len);
  };
  Px v0 = load(0), v1 = load(1), v2 = load(2);
  stage_px(a, ring, 0, v0, len, lane);
  stage_px(a, ring, 1, v1, len - kBatch, lane);
  const int nb = (len + kBatch - 1) / kBatch;
  const int side = p == 1 ? (BWD ? W - 1 : 0) : (BWD ? 0 : W - 1);  // where paths 1 and 3 start a new line
  const int xn = BWD ? 1 : W - 2;                                   // column c-1
  uint16_t* cs = a.cs[BWD ? 1 : 0];
  uint16_t* cs_min = a.cs_min[BWD ? 1 : 0];
  for (int b = 0; b < nb; b++) {
    cp_async_wait<1>();
    __syncwarp();  // the batch's costs are every lane's
    const int n = min(kBatch, len - b * kBatch);
#pragma unroll 1
    for (int i = 0; i < n; i++) {
      if ((p & 1) && x == side && b + i > 0) state_init(s, lane);
      const Range g(__shfl_sync(0xffffffffu, v0.qc, i));
      const uint32_t off8 = __shfl_sync(0xffffffffu, v0.off8, i), pw = __shfl_sync(0xffffffffu, v0.p2, i);
      const uint32_t P2 = (p & 1) ? pw >> 16 : pw & 0xffffu;
      const uint8_t* rawp = ring_slot(a, ring, b, i);
      ragged_step(s, g, BWD ? p2prev : P2, rawp, a, lane);
      p2prev = P2;
      ragged_add(s, g, a.agg + (size_t)off8 * 8, false, rawp, lane);
      if (p < 2 && x == xn) state_put(a, cs, cs_min, (size_t)(BWD ? H - 1 - y : y) * 2 + p, s, lane);
      if (!BWD && p > 0 && y == a.y_b) state_put(a, a.edge, a.edge_min, (size_t)(p - 1) * W + x, s, lane);
      x += dx;
      y += dy;
      if ((unsigned)x >= (unsigned)W) {
        x -= dx * W;
        y += turn;
      }
    }
    __syncwarp();  // every lane has read them before they are replaced
    v0 = v1;
    v1 = v2;
    stage_px(a, ring, b + 2, v1, len - (b + 2) * kBatch, lane);
    v2 = load(b + 3);
  }
  cp_async_wait<0>();
}

// Paths 0 and 1 of a pass's revisits R(c, y), a warp each.
template <bool BWD>
__global__ void __launch_bounds__(64) k_ragged_revisit(const RagArgs a) {
  extern __shared__ __align__(16) uint8_t smem_ragged[];
  const int lane = threadIdx.x & 31, k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (k >= a.n_rev[BWD ? 1 : 0]) return;
  uint8_t* ring = smem_ragged + (size_t)(threadIdx.x >> 5) * warp_smem(a.rounds, a.ring_bytes);
  RState s;
  state_new(s, a, reinterpret_cast<uint16_t*>(ring + 2 * kBatch * a.ring_bytes), lane);
  const int W = a.W, H = a.H;
  const int* sch = a.sched[BWD ? 1 : 0];
  const int y = sch[3 * H + k], xc = BWD ? 0 : W - 1, xn = BWD ? 1 : W - 2;
  auto row = [&](int t) { return BWD ? H - 1 - t : t; };
  const uint4 inf = __ldg(a.info + (size_t)row(y) * W + xc);
  const Range g(inf.y);
  for (int o = lane; o < g.cap / 8; o += 32)
    *reinterpret_cast<uint2*>(ring + kPad + o * 8) = __ldg(reinterpret_cast<const uint2*>(a.raw + ((size_t)inf.x + o) * 8));
  __syncwarp();
#pragma unroll 1
  for (int p = 0; p < 2; p++) {
    const int e = sch[p * H + y], kind = src_kind(e);
    uint32_t p2 = 0;
    state_init(s, lane);
    if (kind == kSrcEdge) {
      if (a.y_b >= 0) {
        state_get(a, a.edge, a.edge_min, xn, s, lane);
        p2 = p2_between(a, xc, row(y), xn, a.y_b);
      }
    } else if (kind != kSrcInit) {
      state_get(a, a.cs[BWD ? 1 : 0], a.cs_min[BWD ? 1 : 0], (size_t)src_row(e) * 2 + (kind - kSrcCs), s, lane);
      p2 = p2_between(a, xc, row(y), xn, row(src_row(e)));
    }
    ragged_step(s, g, p2, ring, a, lane);
    ragged_add(s, g, a.agg + (size_t)inf.x * 8, false, ring, lane);
    // R(y_b) is what pass -1 will read at the last column
    if (!BWD && p == 1 && (sch[2 * H + y] & 1)) state_put(a, a.edge, a.edge_min, xc, s, lane);
  }
}

// The per-pixel table of the walks: P2 is that of pass +1's paths (pass -1 crosses the same edges the other way).
__global__ void k_ragged_info(const RagArgs a, const uint16_t* __restrict__ start, const uint16_t* __restrict__ cap,
                              const uint64_t* __restrict__ off, int min_lo, uint4* __restrict__ info) {
  const int pi = blockIdx.x * blockDim.x + threadIdx.x;
  if (pi >= a.W * a.H) return;
  const int y = pi / a.W, x = pi - y * a.W;
  uint32_t v[4];
#pragma unroll
  for (int p = 0; p < 4; p++) {
    const int xn = x + (p < 2 ? -1 : p == 2 ? 0 : 1), yn = p == 0 ? y : y - 1;
    v[p] = xn >= 0 && xn < a.W && yn >= 0 ? p2_between(a, x, y, xn, yn) : 0u;  // outside: never used (the line starts there)
  }
  info[pi] = make_uint4((uint32_t)(off[pi] >> 3), (uint32_t)(start[pi] - min_lo) | (uint32_t)cap[pi] << 16, v[0] | v[1] << 16, v[2] | v[3] << 16);
}

__global__ void k_ragged_check(const uint16_t* __restrict__ start, const uint16_t* __restrict__ cap, int W, int H, int min_lo, int max_hi,
                               int* flag) {
  const int pi = blockIdx.x * blockDim.x + threadIdx.x;
  if (pi >= W * H) return;
  const int q = start[pi] - min_lo, c = cap[pi];
  bool bad = q < 0 || c == 0 || (c & 7) || q + c > max_hi + 7;
  if (!bad && q + c > max_hi) {
    const int y = pi / W, x = pi - y * W;
    bad = x < 2 || y < 2 || x >= W - 2 || y >= H - 2;
    for (int dy = -2; dy <= 2 && !bad; dy++)
      for (int dx = -2; dx <= 2; dx++) bad |= start[pi + dy * W + dx] - min_lo <= 7;
  }
  if (bad) *flag = 1;
}

struct RaggedLayout {
  size_t info, edge, edge_min, cs, cs_min, sched, total;
};
int rounds_of(int max_hi) { return (max_hi + 9 + kRound - 1) / kRound; }
RaggedLayout ragged_layout(int W, int H, int max_hi) {
  auto al = [](size_t v) { return (v + 255) & ~(size_t)255; };
  const size_t st = (size_t)rounds_of(max_hi) * kRound * 2;
  RaggedLayout s;
  size_t o = 0;
  s.info = o; o += al((size_t)W * H * 16);
  s.edge = o; o += al((size_t)3 * W * st);
  s.edge_min = o; o += al((size_t)3 * W * 2);
  s.cs = o; o += al((size_t)2 * H * 2 * st);
  s.cs_min = o; o += al((size_t)2 * H * 2 * 2);
  s.sched = o; o += al((size_t)2 * 4 * H * 4);
  s.total = o;
  return s;
}

}  // namespace

void launch_ragged_check(const LayerGeom& g, int* flag, cudaStream_t s) {
  cudaMemsetAsync(flag, 0, sizeof(int), s);
  k_ragged_check<<<(g.W * g.H + 255) / 256, 256, 0, s>>>(g.start, g.cap, g.W, g.H, g.min_lo, g.max_hi, flag);
  count_launches(1);
}

// Layers this form takes (besides the device's check): even tiles (a row's half of the line buffer is its parity), the
// no-saturation bound of the uniform forms (P2 up to 1744), at most 887 planes, offsets that fit the table's 32 bits.
bool ragged_lines_supported(int W, int H, int tile, uint16_t p1, float p2scale, int max_hi, uint64_t volume) {
  volatile float p1f = (float)p1;
  const float p2base = p1f * p2scale;
  return W >= 3 && H >= 2 && (tile & 1) == 0 && tile >= 2 && p2scale >= 0.0f && p2base <= 1744.0f && p1 <= 60000 &&
         rounds_of(max_hi) <= kMaxRounds && (uint64_t)W * H < (1ull << 29) && volume < (1ull << 35);
}
size_t ragged_lines_scratch_bytes(int W, int H, int max_hi) { return ragged_layout(W, H, max_hi).total; }

// agg must hold zeros.
int run_ragged_lines(const LayerGeom& g, uint16_t p1, float p2scale, const float gw[4], const uint8_t* raw, uint16_t* agg, void* scratch,
                     size_t scratch_bytes, cudaStream_t s) {
  const int W = g.W, H = g.H;
  const RaggedLayout L = ragged_layout(W, H, g.max_hi);
  if (scratch_bytes < L.total) return 9;
  char* base = static_cast<char*>(scratch);
  RagArgs a;
  std::memset(&a, 0, sizeof a);
  std::vector<int> host((size_t)2 * 4 * H, 0);
  int* dsched = reinterpret_cast<int*>(base + L.sched);
  const size_t st = (size_t)rounds_of(g.max_hi) * kRound;
  for (int pass = 0; pass < 2; pass++) {
    RevisitSchedule sch;
    build_revisit_schedule(W, H, g.tile, pass == 1, sch);
    if (pass == 0) a.y_b = sch.y_b;
    int* h = host.data() + (size_t)pass * 4 * H;
    const std::vector<int>* cols[3] = {&sch.src0, &sch.src1, &sch.extra};
    for (int k = 0; k < 3; k++) std::memcpy(h + (size_t)k * H, cols[k]->data(), (size_t)H * 4);
    int* rl = h + (size_t)3 * H;
    for (int y = 0; y < H; y++)
      for (int k = 0; k < sch.batch_count[y]; k++) rl[a.n_rev[pass]++] = sch.batch_first[y] + k;
    for (int k = 0; k < sch.end_count; k++) rl[a.n_rev[pass]++] = sch.end_first + k;
    a.sched[pass] = dsched + (size_t)pass * 4 * H;
    a.cs[pass] = reinterpret_cast<uint16_t*>(base + L.cs) + (size_t)pass * H * 2 * st;
    a.cs_min[pass] = reinterpret_cast<uint16_t*>(base + L.cs_min) + (size_t)pass * H * 2;
  }
  if (cudaMemcpyAsync(dsched, host.data(), host.size() * 4, cudaMemcpyHostToDevice, s) != cudaSuccess) return 10;
  a.W = W; a.H = H; a.T = g.tile;
  a.raw = raw; a.agg = agg; a.guidance = g.guidance;
  a.p1x2 = (uint32_t)p1 * 0x10001u;
  a.one = 1;
  volatile float p1f = (float)p1;
  a.p2base = p1f * p2scale;
  for (int i = 0; i < 4; i++) a.gw[i] = gw[i];
  a.edge = reinterpret_cast<uint16_t*>(base + L.edge);
  a.edge_min = reinterpret_cast<uint16_t*>(base + L.edge_min);
  a.ring_bytes = ring_bytes_of(g.max_hi);
  uint4* info = reinterpret_cast<uint4*>(base + L.info);
  a.info = info;
  k_ragged_info<<<(W * H + 255) / 256, 256, 0, s>>>(a, g.start, g.cap, g.off, g.min_lo, info);
  count_launches(1);
  a.rounds = rounds_of(g.max_hi);
  const int blocks = (1 + 3 * W + H + 1) / 2, smem = 2 * warp_smem(a.rounds, a.ring_bytes);
  // (a kernel's limit is one for all threads of the process: another one's smaller layer must not lower it before this launch)
  static_assert(2 * warp_smem(kMaxRounds, ring_bytes_of(kMaxRounds * kRound - 9)) <= 48 * 1024, "within every kernel's default limit");
  k_ragged_pass<false><<<blocks, 64, smem, s>>>(a);
  if (a.n_rev[0]) k_ragged_revisit<false><<<(a.n_rev[0] + 1) / 2, 64, smem, s>>>(a);
  k_ragged_pass<true><<<blocks, 64, smem, s>>>(a);
  if (a.n_rev[1]) k_ragged_revisit<true><<<(a.n_rev[1] + 1) / 2, 64, smem, s>>>(a);
  count_launches(2 + (a.n_rev[0] > 0) + (a.n_rev[1] > 0));
  return 0;
}

}  // namespace lux
