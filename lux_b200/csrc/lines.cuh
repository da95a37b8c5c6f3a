// What walks along single lines share (sgm_lines.cu, census_sgm.cu): the lines of a path, a lane's planes and the step.
#pragma once
#include "common.cuh"
#include "sgm_paths.cuh"

namespace lux {

namespace {

constexpr int kSeg = 8;  // pixels of a segment: the forward states kept, and the aggregates staged in shared memory

#define kPastRaw make_uint2(0xffffffffu, 0xffffffffu)  // the raw costs of lanes past the planes
struct L4 {  // eight planes of a lane
  uint32_t r[4];
};

// One path step of a line (DenseStereoSgm.cs:276-313), state in place: L and its minimum md in both halves. p2d: P2 in both
// halves. first / last: the line's lanes holding plane 0 and plane n-1 (BEYOND lies beyond). Lanes past the last one hold raw
// costs of 255: their L is at least 255 (no step's terms are below md), and the least L of the planes is at most 255 (the
// cheapest plane of the step before costs its raw cost here), so they never make a smaller minimum.
// BEYOND: what lies beyond the planes; a: the penalty p1x2 and the multiplier one.
template <int GL, uint32_t BEYOND = kInit2, class Args>
LUX_DEV void line_step(L4& L, uint32_t& md, const L4& raw2, uint32_t p2d, const Args& a, bool first, bool last) {
  const uint32_t one = a.one, neg = 0u - a.one;
  uint32_t prev = __shfl_up_sync(0xffffffffu, L.r[3], 1, GL);
  uint32_t next = __shfl_down_sync(0xffffffffu, L.r[0], 1, GL);
  if (first) prev = BEYOND;
  if (last) next = BEYOND;
  const uint32_t p2x = p2d * one + md;
  const uint32_t lo = __byte_perm(prev, L.r[3], 0x5432), hi = __byte_perm(L.r[0], next, 0x5432);  // planes (-1, 3) and (4, 8)
  const uint32_t t0 = vmin2(vmin2(vmin2(lo, L.r[1]) * one + a.p1x2, L.r[0]), p2x);
  const uint32_t t1 = vmin2(vmin2(vmin2(L.r[0], L.r[2]) * one + a.p1x2, L.r[1]), p2x);
  const uint32_t t2 = vmin2(vmin2(vmin2(L.r[1], L.r[3]) * one + a.p1x2, L.r[2]), p2x);
  const uint32_t t3 = vmin2(vmin2(vmin2(L.r[2], hi) * one + a.p1x2, L.r[3]), p2x);
  L.r[0] = t0 * one + (md * neg + raw2.r[0]);
  L.r[1] = t1 * one + (md * neg + raw2.r[1]);
  L.r[2] = t2 * one + (md * neg + raw2.r[2]);
  L.r[3] = t3 * one + (md * neg + raw2.r[3]);
  uint32_t m = vmin2(vmin2(L.r[0], L.r[1]), vmin2(L.r[2], L.r[3]));
  m = vmin2(m, __byte_perm(m, 0, 0x1032));
  if constexpr (GL == 32) {
    md = __reduce_min_sync(0xffffffffu, m);
  } else if constexpr (GL == 16) {  // two whole-warp reductions wait less than four shuffles: census walks of 16 lanes 3.48 -> 3.04 ms
    const bool up = threadIdx.x & 16;
    const uint32_t m0 = __reduce_min_sync(0xffffffffu, up ? 0xffffffffu : m), m1 = __reduce_min_sync(0xffffffffu, up ? m : 0xffffffffu);
    md = up ? m1 : m0;
  } else {
#pragma unroll
    for (int o = GL / 2; o > 0; o >>= 1) m = vmin2(m, __shfl_xor_sync(0xffffffffu, m, o));
    md = m;
  }
}

LUX_DEV void unpack8(L4& v, uint2 b) {  // raw costs of a lane's planes
  const uint32_t e = __byte_perm(b.x, b.y, 0x5410), f = __byte_perm(b.x, b.y, 0x7632);
  v.r[0] = e & 0x00ff00ffu;
  v.r[1] = (e >> 8) & 0x00ff00ffu;
  v.r[2] = f & 0x00ff00ffu;
  v.r[3] = (f >> 8) & 0x00ff00ffu;
}
LUX_DEV uint4 as_uint4(const L4& v) { return make_uint4(v.r[0], v.r[1], v.r[2], v.r[3]); }
LUX_DEV L4 as_l4(uint4 t) { return L4{{t.x, t.y, t.z, t.w}}; }

// The raw costs of a walk's next steps, staged by cp.async in batches of kBatch steps: two batch buffers in shared memory a
// warp, 8 bytes a lane and step. While one batch is walked the next is in flight (a register queue of loads would be
// waited for in full at every step: the scoreboards of a warp do not count that many loads apart).
constexpr int kBatch = 8;
struct RawRing {
  uint2* base;  // this lane's slot of step 0
  LUX_DEV RawRing(uint2* slot0, bool in) : base(slot0) {
    if (!in)
      for (int i = 0; i < 2 * kBatch; i++) base[i * 32] = kPastRaw;
  }
  LUX_DEV void stage(int b, int i, const uint8_t* src) { cp_async8(base + ((b & 1) * kBatch + i) * 32, src); }
  LUX_DEV uint2 get(int b, int i) const { return base[((b & 1) * kBatch + i) * 32]; }
};

// The lines of path p: line r is the pixels r, r + step, r + 2·step, ... (path 0: row r from its first pixel).
LUX_DEV int line_step_of(int p, int W) { return p == 0 ? 1 : p == 1 ? W + 1 : p == 2 ? W : W - 1; }
template <class Args>  // (with the image's size W, H)
LUX_DEV int line_count(const Args& a, int p) {  // (no line without pixels: a single row has no pixel W)
  return p == 0 ? a.H : p == 1 ? min(a.W + 1, a.W * a.H) : line_step_of(p, a.W);
}
template <class Args>
LUX_DEV int line_first(const Args& a, int p, int r) { return p == 0 ? r * a.W : r; }
template <class Args>
LUX_DEV int line_len(const Args& a, int p, int r) {
  return p == 0 ? a.W : p == 2 ? a.H : (a.W * a.H - r + line_step_of(p, a.W) - 1) / line_step_of(p, a.W);
}
// A walk's pixel at the start of a batch, with its column (kept for paths 1 and 3, which restart at the sides). dx: the
// column's change a step.
struct Walk {
  int pi, x, step, dx, W;
  LUX_DEV void advance() {
    pi += step * kBatch;
    x += dx * kBatch;
    if ((unsigned)x >= (unsigned)W) x -= dx * W;
  }
};
template <class Args>
LUX_DEV Walk walk_at(const Args& a, int p, int pi, int dir) {
  Walk w;
  w.pi = pi;
  w.W = a.W;
  w.step = dir * line_step_of(p, a.W);
  w.dx = p == 1 ? dir : p == 3 ? -dir : 0;
  w.x = w.dx ? pi % a.W : 0;
  return w;
}
// Stages a batch of a line's raw costs (len of them, n planes a pixel) for the lane.
LUX_DEV void stage_batch(RawRing& rr, int b, const uint8_t* raw, int n, const Walk& w, int len, int gl, bool in) {
  if (in) {
    const uint8_t* src = raw + (size_t)w.pi * n + gl * 8;
    const long long ds = (long long)w.step * n;
#pragma unroll
    for (int i = 0; i < kBatch; i++, src += ds)
      if (i < len) rr.stage(b, i, src);
  }
  cp_async_commit();
}

// The winner-take-all of every pixel: the first plane of the least aggregate (DenseStereoSgm.cs:228-230).
template <int GL>
LUX_DEV int wta_line(const L4& s, int gl, int lane, bool in) {
  const uint32_t m = vmin2(vmin2(s.r[0], s.r[1]), vmin2(s.r[2], s.r[3]));
  const uint32_t lm = in ? min(m & 0xffffu, m >> 16) : 0xffffffffu;
  uint32_t best = lm;
  if constexpr (GL == 32) {
    best = __reduce_min_sync(0xffffffffu, lm);
  } else {
#pragma unroll
    for (int o = GL / 2; o > 0; o >>= 1) best = min(best, __shfl_xor_sync(0xffffffffu, best, o));
  }
  const uint32_t votes = __ballot_sync(0xffffffffu, lm == best) >> (lane - gl) & (GL == 32 ? 0xffffffffu : (1u << (GL & 31)) - 1u);
  // the first of the lane's planes that equals best (meant for the winning lane): bit k (planes 0..3) or 16 + k (4..7) of
  // `above` says whether plane k is above it
  const uint32_t best2 = best * 0x10001u, one2 = 0x00010001u;
  const uint32_t above = vmin2(s.r[0] - best2, one2) + vmin2(s.r[1] - best2, one2) * 2u + vmin2(s.r[2] - best2, one2) * 4u +
                         vmin2(s.r[3] - best2, one2) * 8u;
  const int bit = __ffs(~above & 0x000f000fu) - 1, win = __ffs(votes) - 1;
  const int k = (bit & 3) + ((bit & 16) >> 2);
  return win * 8 + __shfl_sync(0xffffffffu, k, win, GL);
}

}  // namespace

}  // namespace lux
