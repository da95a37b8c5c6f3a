// What walks along single lines share (sgm_lines.cu, census_sgm.cu): the lines of a path, a lane's planes and the step.
#pragma once
#include "common.cuh"
#include "sgm_paths.cuh"

namespace lux {

namespace {

constexpr int kSeg = 8;  // pixels of a segment: the forward states kept, and the aggregates staged in shared memory

// K planes p0..p(K-1) of a lane (8, or 4 where lines are few) as u16 pairs (p0, pK/2), (p1, pK/2+1), ...
template <int K>
struct Planes {
  uint32_t r[K / 2];
};
using L4 = Planes<8>;
// The lane's raw costs as they are loaded, and those of lanes past the planes.
template <int K>
struct RawOf;
template <>
struct RawOf<8> {
  using type = uint2;
  static LUX_DEV uint2 past() { return make_uint2(0xffffffffu, 0xffffffffu); }
};
template <>
struct RawOf<4> {
  using type = uint32_t;
  static LUX_DEV uint32_t past() { return 0xffffffffu; }
};
#define kPastRaw RawOf<8>::past()

// One path step of a line (DenseStereoSgm.cs:276-313), state in place: L and its minimum md in both halves. p2d: P2 in both
// halves. first / last: the line's lanes holding plane 0 and plane n-1 (BEYOND lies beyond). Lanes past the last one hold raw
// costs of 255: their L is at least 255 (no step's terms are below md), and the least L of the planes is at most 255 (the
// cheapest plane of the step before costs its raw cost here), so they never make a smaller minimum.
// BEYOND: what lies beyond the planes; a: the penalty p1x2 and the multiplier one.
template <int GL, uint32_t BEYOND = kInit2, int K, class Args>
LUX_DEV void line_step(Planes<K>& L, uint32_t& md, const Planes<K>& raw2, uint32_t p2d, const Args& a, bool first, bool last) {
  constexpr int N = K / 2;
  const uint32_t one = a.one, neg = 0u - a.one;
  uint32_t prev = __shfl_up_sync(0xffffffffu, L.r[N - 1], 1, GL);
  uint32_t next = __shfl_down_sync(0xffffffffu, L.r[0], 1, GL);
  if (first) prev = BEYOND;
  if (last) next = BEYOND;
  const uint32_t p2x = p2d * one + md;
  const uint32_t lo = __byte_perm(prev, L.r[N - 1], 0x5432), hi = __byte_perm(L.r[0], next, 0x5432);  // planes (-1, N - 1) and (N, K)
  uint32_t t[N];
#pragma unroll
  for (int i = 0; i < N; i++)
    t[i] = vmin2(vmin2(vmin2(i == 0 ? lo : L.r[i > 0 ? i - 1 : 0], i == N - 1 ? hi : L.r[i < N - 1 ? i + 1 : 0]) * one + a.p1x2, L.r[i]), p2x);
#pragma unroll
  for (int i = 0; i < N; i++) L.r[i] = t[i] * one + (md * neg + raw2.r[i]);
  uint32_t m = L.r[0];
  if constexpr (N == 2) m = vmin2(m, L.r[1]);
  else m = vmin2(vmin2(m, L.r[1]), vmin2(L.r[2], L.r[3]));
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

LUX_DEV void unpack(L4& v, uint2 b) {  // raw costs of a lane's planes
  const uint32_t e = __byte_perm(b.x, b.y, 0x5410), f = __byte_perm(b.x, b.y, 0x7632);
  v.r[0] = e & 0x00ff00ffu;
  v.r[1] = (e >> 8) & 0x00ff00ffu;
  v.r[2] = f & 0x00ff00ffu;
  v.r[3] = (f >> 8) & 0x00ff00ffu;
}
LUX_DEV void unpack(Planes<4>& v, uint32_t b) {
  v.r[0] = b & 0x00ff00ffu;
  v.r[1] = (b >> 8) & 0x00ff00ffu;
}
LUX_DEV uint4 as_uint4(const L4& v) { return make_uint4(v.r[0], v.r[1], v.r[2], v.r[3]); }
LUX_DEV L4 as_l4(uint4 t) { return L4{{t.x, t.y, t.z, t.w}}; }

// The raw costs of a walk's next steps, staged by cp.async in batches of kBatch steps: two batch buffers in shared memory a
// warp, a byte a plane and step. While one batch is walked the next is in flight (a register queue of loads would be
// waited for in full at every step: the scoreboards of a warp do not count that many loads apart).
constexpr int kBatch = 8;
template <int K>
struct RawRing {
  using Raw = typename RawOf<K>::type;
  Raw* base;  // this lane's slot of step 0
  LUX_DEV RawRing(Raw* slot0, bool in) : base(slot0) {
    if (!in)
      for (int i = 0; i < 2 * kBatch; i++) base[i * 32] = RawOf<K>::past();
  }
  LUX_DEV void stage(int b, int i, const uint8_t* src) {
    Raw* dst = base + ((b & 1) * kBatch + i) * 32;
    if constexpr (K == 8) cp_async8(dst, src);
    else cp_async4(dst, src);
  }
  LUX_DEV Raw get(int b, int i) const { return base[((b & 1) * kBatch + i) * 32]; }
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
template <int K>
LUX_DEV void stage_batch(RawRing<K>& rr, int b, const uint8_t* raw, int n, const Walk& w, int len, int gl, bool in) {
  if (in) {
    const uint8_t* src = raw + (size_t)w.pi * n + gl * K;
    const long long ds = (long long)w.step * n;
#pragma unroll
    for (int i = 0; i < kBatch; i++, src += ds)
      if (i < len) rr.stage(b, i, src);
  }
  cp_async_commit();
}

// The winner-take-all of every pixel: the first plane of the least aggregate (DenseStereoSgm.cs:228-230).
template <int GL, int K>
LUX_DEV int wta_line(const Planes<K>& s, int gl, int lane, bool in) {
  constexpr int N = K / 2;
  uint32_t m = s.r[0];
#pragma unroll
  for (int i = 1; i < N; i++) m = vmin2(m, s.r[i]);
  const uint32_t lm = in ? min(m & 0xffffu, m >> 16) : 0xffffffffu;
  uint32_t best = lm;
  if constexpr (GL == 32) {
    best = __reduce_min_sync(0xffffffffu, lm);
  } else {
#pragma unroll
    for (int o = GL / 2; o > 0; o >>= 1) best = min(best, __shfl_xor_sync(0xffffffffu, best, o));
  }
  const uint32_t votes = __ballot_sync(0xffffffffu, lm == best) >> (lane - gl) & (GL == 32 ? 0xffffffffu : (1u << (GL & 31)) - 1u);
  // the first of the lane's planes that equals best (meant for the winning lane): bit i (plane i) or 16 + i (plane N + i) of
  // `above` says whether the plane is above it
  const uint32_t best2 = best * 0x10001u, one2 = 0x00010001u;
  uint32_t above = 0;
#pragma unroll
  for (int i = 0; i < N; i++) above += vmin2(s.r[i] - best2, one2) * (1u << i);
  const int bit = __ffs(~above & (((1u << N) - 1) * 0x10001u)) - 1, win = __ffs(votes) - 1;
  const int k = bit & 16 ? (bit & 15) + N : bit;
  return win * K + __shfl_sync(0xffffffffu, k, win, GL);
}

}  // namespace

}  // namespace lux
