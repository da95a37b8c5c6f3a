// Box filter, guidance, plane ranges from the previous layer, CSR offsets, WTA and the upsample chain.
// Each kernel restates one reference function with its exact operation order (file:line in each comment).
#include <algorithm>
#include <atomic>
#include <cstring>

#include <cub/cub.cuh>

#include "common.cuh"
#include "internal.h"

namespace lux {

static std::atomic<uint64_t> g_launches{0};
void count_launches(int n) { g_launches.fetch_add((uint64_t)n, std::memory_order_relaxed); }
uint64_t kernel_launches() { return g_launches.load(); }

// ---- DenseStereo.BoxFilter3 (DenseStereo.cs:93-159): per channel float(Σ)·(1/(cols·rows)), RNE, saturated ----
// DenseLayer.SkipMask (DenseStereoSgm.cs:65-87), SkipMode 2: the image is cut into 64x64 tiles (the last tile of a row or
// column takes the remainder, nx = w/64 + (64 < 2·(w%64))), each drawing from a fresh default-seeded mt19937; its 2x2
// cells in row order take two draws each, dy then dx, and the cell's pixel (x + dx, y + dy) is computed (0), every
// other pixel skipped (0xff). Tiles start at multiples of 64, so a pixel's cell is (x & ~1, y & ~1) and it is the
// chosen one when its parities are (dx, dy). bits: the stream's low bits (host_skip_stream_bits).
__global__ void k_skip_mask(uint8_t* __restrict__ m, int w, int h, int nx, int ny, const uint32_t* __restrict__ bits) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y;
  if (x >= w || y >= h) return;
  const int i = min(x >> 6, nx - 1), j = min(y >> 6, ny - 1);
  const int x0 = 64 * i, x1 = min(w, x0 + (i == nx - 1 ? 128 : 64)), y0 = 64 * j;
  const int c = ((y - y0) >> 1) * ((x1 - x0 + 1) >> 1) + ((x - x0) >> 1);  // the cell's index in its tile
  const int k = 2 * c;
  const int dy = (__ldg(bits + (k >> 5)) >> (k & 31)) & 1, dx = (__ldg(bits + ((k + 1) >> 5)) >> ((k + 1) & 31)) & 1;
  m[(size_t)y * w + x] = ((x & 1) == dx && (y & 1) == dy) ? 0 : 0xff;
}

void launch_skip_mask(int mode, int w, int h, const uint32_t* bits, uint8_t* m, cudaStream_t s) {
  if (mode == 0) {
    cudaMemsetAsync(m, 0, (size_t)w * h, s);
    return;
  }
  int nx = w / 64 + (64 < 2 * (w % 64) ? 1 : 0), ny = h / 64 + (64 < 2 * (h % 64) ? 1 : 0);
  if (nx < 1) nx = 1;
  if (ny < 1) ny = 1;
  k_skip_mask<<<dim3((w + 255) / 256, h), 256, 0, s>>>(m, w, h, nx, ny, bits);
  count_launches(1);
}

__global__ void k_box_filter3(const uint8_t* __restrict__ src, int w, int h, int stride, uint8_t* __restrict__ dst) {
  int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y;
  if (x >= w) return;
  int y0 = max(y - 1, 0), y1 = min(y + 1, h - 1), x0 = max(x - 1, 0), x1 = min(x + 1, w - 1);
  int rows = y1 - y0 + 1, cols = x1 - x0 + 1;
  // vector form: 1/(2·rows) at the edge columns, 1/(3·rows) inside (:110); the scalar form gives the same divisors
  float inv = __fdiv_rn(1.0f, __fmul_rn((float)cols, (float)rows));
  int s0 = 0, s1 = 0, s2 = 0, s3 = 0;
  for (int yy = y0; yy <= y1; yy++)
    for (int xx = x0; xx <= x1; xx++) {
      uchar4 p = __ldg(reinterpret_cast<const uchar4*>(src) + (size_t)yy * stride + xx);
      s0 += p.x; s1 += p.y; s2 += p.z; s3 += p.w;
    }
  auto q = [&](int s) {
    int v = __float2int_rn(__fmul_rn((float)s, inv));  // cvtps2dq
    return (unsigned char)min(max(v, 0), 255);           // packssdw + packuswb
  };
  reinterpret_cast<uchar4*>(dst)[(size_t)y * w + x] = make_uchar4(q(s0), q(s1), q(s2), q(s3));
}

void launch_box_filter3(const uint8_t* src, int w, int h, int stride, uint8_t* dst, cudaStream_t s) {
  dim3 grid((w + 127) / 128, h);
  k_box_filter3<<<grid, 128, 0, s>>>(src, w, h, stride, dst);
  count_launches(1);
}

// ---- DenseStereo.Guidance (DenseStereo.cs:163-177) ----
__global__ void k_guidance(const uchar4* __restrict__ img0, int w0, int h0, int w, int h, int scale, uchar4* __restrict__ out) {
  int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y;
  if (x >= w) return;
  int sx = x, sy = y;
  if (!(w0 == w && h0 == h)) {
    int half = (scale + (scale >> 31)) >> 1;
    sy = min(scale * y + half, h0 - 1);
    sx = min(scale * x + half, w0 - 1);
  }
  out[(size_t)y * w + x] = img0[(size_t)sy * w0 + sx];
}

void launch_guidance(const uint8_t* img0, int w0, int h0, int w, int h, int scale, uchar4* out, cudaStream_t s) {
  dim3 grid((w + 127) / 128, h);
  k_guidance<<<grid, 128, 0, s>>>(reinterpret_cast<const uchar4*>(img0), w0, h0, w, h, scale, out);
  count_launches(1);
}

// ---- DenseLayer.RangeFromPrevious (DenseStereoSgm.cs:91-140) ----
// scratch: idx[pw*ph], hmin, hmax (u16)
size_t range_from_previous_scratch_bytes(int pw, int ph) { return (size_t)pw * ph * 2 * 3 + 256; }

// plane index of every previous pixel: #{j : b[j] <= rcp(depth)} as the scan `while (c < n && b[c] <= v) c++` (:101)
__global__ void k_plane_index(const float* __restrict__ depth, int npx, const float* __restrict__ b, int n, int monotone,
                              const uint32_t* __restrict__ rcp_table, uint16_t* __restrict__ idx) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= npx) return;
  float v = rcp_approx(depth[i], rcp_table);
  int c;
  if (monotone) {  // b non-decreasing: the first index with !(b[c] <= v) by bisection
    int lo = 0, hi = n;
    while (lo < hi) {
      int mid = (lo + hi) >> 1;
      if (__ldg(b + mid) <= v) lo = mid + 1; else hi = mid;
    }
    c = lo;
  } else {
    c = 0;
    while (c < n && __ldg(b + c) <= v) c++;
  }
  idx[i] = (uint16_t)c;
}

// 4-wide horizontal min/max over computed pixels x-1..x+2 (clamped) (:105-117)
__global__ void k_hminmax(const uint16_t* __restrict__ idx, const uint8_t* __restrict__ skip, int pw, int ph, uint16_t* __restrict__ hmin,
                          uint16_t* __restrict__ hmax) {
  int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y;
  if (x >= pw) return;
  unsigned mn = 0xffff, mx = 0;
  for (int k = -1; k <= 2; k++) {
    int xx = min(max(x + k, 0), pw - 1);
    if (skip[(size_t)y * pw + xx] > 0) continue;
    unsigned v = idx[(size_t)y * pw + xx];
    mn = min(mn, v);
    mx = max(mx, v);
  }
  hmin[(size_t)y * pw + x] = (uint16_t)mn;
  hmax[(size_t)y * pw + x] = (uint16_t)mx;
}

// vertical 4-tall min/max (:118-125) sampled at the nearest previous pixel, margin, range (:126-138)
__global__ void k_ranges(const uint16_t* __restrict__ hmin, const uint16_t* __restrict__ hmax, int pw, int ph, int W, int H, float fx,
                         float fy, int n, int margin, uint16_t* __restrict__ start, uint16_t* __restrict__ count, int* minmax) {
  int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y;
  int lo = 0x7fffffff, hi = 0;
  if (x < W) {
    int py = f2i(__fmul_rn((float)y, fy)), px = f2i(__fmul_rn((float)x, fx));
    py = min(max(py, 0), ph - 1);  // (float)y·fy never leaves [0, ph-1]; the clamp only guards the load
    px = min(max(px, 0), pw - 1);
    unsigned mn = 0xffff, mx = 0;
    for (int k = -1; k <= 2; k++) {
      int yy = min(max(py + k, 0), ph - 1);
      mn = min(mn, (unsigned)hmin[(size_t)yy * pw + px]);
      mx = max(mx, (unsigned)hmax[(size_t)yy * pw + px]);
    }
    lo = max(0, (int)mn - margin);
    hi = min(n - 1, (int)mx + 1);
    size_t i = (size_t)y * W + x;
    start[i] = (uint16_t)lo;
    count[i] = (uint16_t)(hi - lo);
    lo &= 0xffff;
    hi &= 0xffff;
  }
  // block reduction, then one atomic per block
  for (int o = 16; o > 0; o >>= 1) {
    lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
  if ((threadIdx.x & 31) == 0) {
    atomicMin(&minmax[0], lo);
    atomicMax(&minmax[1], hi);
  }
}

void launch_range_from_previous(const float* prev_depth, const uint8_t* prev_skip, int pw, int ph, const float* b, int monotone,
                                int n, const uint32_t* rcp_table, int W, int H, int margin, uint16_t* start, uint16_t* count,
                                int* minmax, void* scratch, cudaStream_t s) {
  uint16_t* idx = static_cast<uint16_t*>(scratch);
  uint16_t* hmin = idx + (size_t)pw * ph;
  uint16_t* hmax = hmin + (size_t)pw * ph;
  int npx = pw * ph;
  k_plane_index<<<(npx + 255) / 256, 256, 0, s>>>(prev_depth, npx, b, n, monotone, rcp_table, idx);
  count_launches(1);
  dim3 g1((pw + 127) / 128, std::min(ph, 65535));
  k_hminmax<<<g1, 128, 0, s>>>(idx, prev_skip, pw, ph, hmin, hmax);
  count_launches(1);
  float fy = (float)(ph - 1) / (float)(H - 1), fx = (float)(pw - 1) / (float)(W - 1);
  dim3 g2((W + 127) / 128, H);
  k_ranges<<<g2, 128, 0, s>>>(hmin, hmax, pw, ph, W, H, fx, fy, n, margin, start, count, minmax);
  count_launches(1);
}

// ---- caps and CSR offsets (DenseStereoSgm.cs:53-58): cap = count rounded up to align ----
__global__ void k_caps(const uint16_t* __restrict__ count, int npx, int align, uint16_t* __restrict__ cap, uint64_t* __restrict__ c64) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= npx) return;
  int c = ((count[i] + align - 1) / align) * align;
  cap[i] = (uint16_t)c;
  c64[i] = (uint64_t)c;
}

size_t caps_offsets_scratch_bytes(int npx) {
  size_t tmp = 0;
  cub::DeviceScan::ExclusiveSum(nullptr, tmp, (const uint64_t*)nullptr, (uint64_t*)nullptr, npx + 1);
  return tmp + (size_t)(npx + 1) * 8 + 256;
}

void launch_caps_offsets(const uint16_t* count, int npx, int align, uint16_t* cap, uint64_t* off, void* scratch, size_t scratch_bytes,
                         cudaStream_t s) {
  uint64_t* c64 = static_cast<uint64_t*>(scratch);
  void* tmp = static_cast<char*>(scratch) + ((size_t)(npx + 1) * 8 + 255) / 256 * 256;
  size_t tmp_bytes = scratch_bytes - ((size_t)(npx + 1) * 8 + 255) / 256 * 256;
  cudaMemsetAsync(c64 + npx, 0, 8, s);
  k_caps<<<(npx + 255) / 256, 256, 0, s>>>(count, npx, align, cap, c64);
  count_launches(1);
  cub::DeviceScan::ExclusiveSum(tmp, tmp_bytes, c64, off, npx + 1, s);
}

// Σ (8 + cap·(skipped ? 2 : 3)) of DenseLayer.MemoryEstimate (DenseStereoSgm.cs:153)
__global__ void k_estimate(const uint16_t* __restrict__ count, const uint8_t* __restrict__ skip, int npx, int align,
                           unsigned long long* out) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  unsigned long long v = 0;
  if (i < npx) {
    int c = ((count[i] + align - 1) / align) * align;
    v = 8ull + (unsigned long long)c * (skip[i] == 0 ? 3ull : 2ull);
  }
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0 && v) atomicAdd(out, v);
}

void launch_estimate_terms(const uint16_t* count, const uint8_t* skip, int npx, int align, unsigned long long* out, cudaStream_t s) {
  k_estimate<<<(npx + 255) / 256, 256, 0, s>>>(count, skip, npx, align, out);
  count_launches(1);
}

// A pixel whose cap is not a multiple of 8 makes the reference's scalar SGM lanes write agg[cap] (DenseStereoSgm.cs:302-311).
__global__ void k_check_caps(const uint16_t* __restrict__ cap, int npx, int* err) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < npx && cap[i] != 0 && (cap[i] & 7) != 0) atomicCAS(err, 0, 7 /* LUX_ERR_INDEX */);
}
void launch_check_caps(const uint16_t* cap, int npx, int* err, cudaStream_t s) {
  k_check_caps<<<(npx + 255) / 256, 256, 0, s>>>(cap, npx, err);
  count_launches(1);
}

// A grey image of `bits` per sample (9..16, u16) as the reference's grey YUVA bytes (Y, 128, 128, 255): Y = (v + half) >>
// (bits - 8) saturated at 255, half = 1 << (bits - 9) (12-bit: (v + 8) >> 4). Four pixels a thread.
__global__ void k_grey16_to_rgba8(const uint16_t* __restrict__ src, int w, int h, int stride, int bits, uchar4* __restrict__ dst) {
  const int shift = bits - 8, half = 1 << (shift - 1);
  const int x4 = (blockIdx.x * blockDim.x + threadIdx.x) * 4, y = blockIdx.y;
  if (x4 >= w || y >= h) return;
  const uint16_t* row = src + (size_t)y * stride;
  uchar4* out = dst + (size_t)y * w;
  for (int k = 0; k < 4 && x4 + k < w; k++) {
    const int v = min(255, ((int)row[x4 + k] + half) >> shift);
    out[x4 + k] = make_uchar4((unsigned char)v, 128, 128, 255);
  }
}
void launch_grey16_to_rgba8(const uint16_t* src, int w, int h, int stride, int bits, uint8_t* dst, cudaStream_t s) {
  dim3 grid((w + 4 * 128 - 1) / (4 * 128), h);
  k_grey16_to_rgba8<<<grid, 128, 0, s>>>(src, w, h, stride, bits, reinterpret_cast<uchar4*>(dst));
  count_launches(1);
}

__global__ void k_fill_u16(uint16_t* p, size_t n, uint16_t v) {
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  size_t stride = (size_t)gridDim.x * blockDim.x;
  for (; i < n; i += stride) p[i] = v;
}
void launch_fill_u16(uint16_t* p, size_t n, uint16_t v, cudaStream_t s) {
  if (n == 0) return;
  size_t nb = (n + 255) / 256;
  int blocks = (int)(nb < 148 * 16 ? nb : 148 * 16);
  k_fill_u16<<<blocks, 256, 0, s>>>(p, n, v);
  count_launches(1);
}

// a first layer: Start 0, Count = Cap = n (DenseStereoSgm.cs:43-46)
__global__ void k_uniform_ranges(uint16_t* start, uint16_t* count, uint16_t* cap, uint64_t* off, int npx, int n) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i > npx) return;
  off[i] = (uint64_t)i * (uint64_t)n;
  if (i == npx) return;
  start[i] = 0;
  count[i] = (uint16_t)n;
  cap[i] = (uint16_t)n;
}
void launch_uniform_ranges(uint16_t* start, uint16_t* count, uint16_t* cap, uint64_t* off, int npx, int n, cudaStream_t s) {
  k_uniform_ranges<<<(npx + 1 + 255) / 256, 256, 0, s>>>(start, count, cap, off, npx, n);
  count_launches(1);
}

// ---- WTA (DenseStereoSgm.cs:225-231): first minimum of agg[0, count) -> Planes[(ushort)(Start + arg)] ----
__global__ void k_wta(const uint16_t* __restrict__ agg, const uint64_t* __restrict__ off, const uint16_t* __restrict__ start,
                      const uint16_t* __restrict__ count, const float* __restrict__ planes, int n, int npx, float* __restrict__ depth,
                      int* err) {
  int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (warp >= npx) return;
  const uint16_t* a = agg + off[warp];
  int cnt = count[warp];
  int best = 0xffff, arg = 0x7fffffff;
  for (int k = lane; k < cnt; k += 32) {
    int v = a[k];
    if (v < best) { best = v; arg = k; }
  }
  for (int o = 16; o > 0; o >>= 1) {
    int ob = __shfl_xor_sync(0xffffffffu, best, o), oa = __shfl_xor_sync(0xffffffffu, arg, o);
    if (ob < best || (ob == best && oa < arg)) { best = ob; arg = oa; }
  }
  if (lane == 0) {
    if (arg == 0x7fffffff) arg = 0;
    int pl = (uint16_t)(start[warp] + arg);
    if (pl >= n) { atomicCAS(err, 0, 7); pl = 0; }
    depth[warp] = planes[pl];
  }
}

void launch_wta(const LayerGeom& g, const uint16_t* agg, float* depth, int* err, cudaStream_t s) {
  int npx = g.W * g.H;
  k_wta<<<(npx + 7) / 8, 256, 0, s>>>(agg, g.off, g.start, g.count, g.planes, g.n_planes, npx, depth, err);
  count_launches(1);
}

// ---- DenseUpsampleLayer (DenseUpsampleLayer.cs:35-218) ----

// g2(x,y) = ImageShift(guide, 0.5, 0.5)(sx, sy) with the 16.16 nearest steps of NearestResize (:69-131): the shifted guide is
// only ever read at these positions, so only they are computed. CubicTap (:56-62) of the half-pixel shift is exactly
// (-1, 9, 9, -1) / 16 in both directions, so every product and sum of the two float passes is a multiple of 1/256 below 2^10,
// exact in any order: they run on integers here, two channels a register vertically, and are rounded once (to even, as cvtps).
// Bound by issue (some 200 operations a pixel): 2080x1560 of a 4160x3120 guide in 32 us; the float passes on byte loads took
// 62 us, on word loads 56. WORDS: the guide's pixels are 4-byte aligned.
template <bool WORDS>
__global__ void __launch_bounds__(128) k_shift_resize(const uint8_t* __restrict__ guide, int gw, int gh, int gstride, int pw, int ph, int stepX,
                                                      int stepY, uint8_t* __restrict__ g2) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  if (x >= pw) return;
  const int sx = (int)((unsigned)stepX * (unsigned)x) >> 16;  // the accumulated xAcc: an int that wraps, past 32767 columns
  int cols[4];
#pragma unroll
  for (int j = 0; j < 4; j++) cols[j] = min(max(sx - 1 + j, 0), gw - 1);  // clamp to edge
  for (int y = blockIdx.y; y < ph; y += gridDim.y) {  // gridDim.y is capped at 65535 rows; taller images loop
    const int sy = (int)((unsigned)stepY * (unsigned)y) >> 16;
    uint32_t px[4][4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const uint8_t* row = guide + (size_t)min(max(sy - 1 + i, 0), gh - 1) * gstride * 4;
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const uint8_t* g = row + (size_t)cols[j] * 4;
        if (WORDS) px[i][j] = __ldg(reinterpret_cast<const uint32_t*>(g));
        else px[i][j] = g[0] | (uint32_t)g[1] << 8 | (uint32_t)g[2] << 16 | (uint32_t)g[3] << 24;
      }
    }
    uint32_t r[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {  // channels h and h + 2
      uint32_t v[4];               // 16 x the column's value + 512, in 0 .. 5102
#pragma unroll
      for (int j = 0; j < 4; j++) {
        auto ch = [&](uint32_t w) { return __byte_perm(w, 0, h ? 0x4341 : 0x4240); };
        v[j] = (ch(px[1][j]) + ch(px[2][j])) * 9u + 0x02000200u - (ch(px[0][j]) + ch(px[3][j]));
      }
      const uint32_t mid = v[1] + v[2], out = v[0] + v[3];
      auto round256 = [](int n) {  // n/256 to the nearest, ties to even: in the low bits of 1.5·2^23 + n/256
        const float f = __fsub_rn(__int_as_float(0x4b400000 + n), 12582912.0f);
        return __float_as_uint(__fmaf_rn(f, 1.0f / 256.0f, 12582912.0f));
      };
      const uint32_t lo = round256((int)((mid & 0xffffu) * 9u - (out & 0xffffu)) - 8192);
      const uint32_t hi = round256((int)((mid >> 16) * 9u - (out >> 16)) - 8192);
      r[h] = __vmins2(__vmaxs2(__byte_perm(lo, hi, 0x5410), 0u), 0x00ff00ffu);
    }
    reinterpret_cast<uint32_t*>(g2)[(size_t)y * pw + x] = r[0] | r[1] << 8;
  }
}

LUX_DEV float up_exp2(float t) {  // Exp2Fast (:151-159)
  const float C1 = __uint_as_float(0x3d9fcb52u), C2 = __uint_as_float(0x3e677e26u), C3 = __uint_as_float(0x3f322226u),
              C4 = __uint_as_float(0x3f7ffb19u);
  t = t < 128.0f ? t : 128.0f;
  t = t > -126.0f ? t : -126.0f;
  int n = f2i(t) + ((int)__float_as_uint(t) >> 31);
  float f = __fsub_rn(t, (float)n);
  float p = __fadd_rn(__fmul_rn(__fadd_rn(__fmul_rn(__fadd_rn(__fmul_rn(f, C1), C2), f), C3), f), C4);
  return __uint_as_float(__float_as_uint(p) + ((unsigned)n << 23));
}
// Two floats a register pair, each operation rounded as its scalar form.
struct F2 {
  uint64_t v;
};
LUX_DEV F2 f2(float a, float b) { F2 r; asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b)); return r; }
LUX_DEV void f2_get(F2 p, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(p.v)); }
LUX_DEV F2 operator+(F2 a, F2 b) { F2 r; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v)); return r; }
LUX_DEV F2 operator*(F2 a, F2 b) { F2 r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v)); return r; }
// a·b for a sum that follows: a pair's mul.rn is contracted with the add.rn that takes its product, in spite of --fmad=false.
// minus0 is (-0.0, -0.0) in a form that the compiler does not see through: a kernel argument.
LUX_DEV F2 mul_alone(F2 a, F2 b, F2 minus0) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(minus0.v));
  return r;
}
LUX_DEV F2 add_up(F2 a, F2 b) { F2 r; asm("add.rp.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v)); return r; }
LUX_DEV F2 f2_neg(F2 a) { return F2{a.v ^ 0x8000000080000000ull}; }

// up_exp2 of two t <= -0.0, given as -t, without conversions: there n = ceil(t) - 1, and t + M rounded up holds ceil(t) in its
// low bits. M = 1.5·2^23 + 511, whose bits end in 511, so a shift of the sum's bits by 23 leaves n alone. t - n is rounded
// once as there: the sum's difference to M + 1 is whole and exact.
LUX_DEV F2 up_exp2_neg(float a, float b, F2 minus0) {
  const float C1 = __uint_as_float(0x3d9fcb52u), C2 = __uint_as_float(0x3e677e26u), C3 = __uint_as_float(0x3f322226u),
              C4 = __uint_as_float(0x3f7ffb19u), M = 12583423.0f;
  const F2 t = f2(-fminf(a, 126.0f), -fminf(b, 126.0f));
  const F2 m = add_up(t, f2(M, M)), f = t + (f2(M + 1.0f, M + 1.0f) + f2_neg(m));
  F2 p = mul_alone(f, f2(C1, C1), minus0) + f2(C2, C2);
  p = mul_alone(p, f, minus0) + f2(C3, C3);
  p = mul_alone(p, f, minus0) + f2(C4, C4);
  float p0, p1, m0, m1;
  f2_get(p, p0, p1);
  f2_get(m, m0, m1);
  return f2(__uint_as_float(__float_as_uint(p0) + (__float_as_uint(m0) << 23)), __uint_as_float(__float_as_uint(p1) + (__float_as_uint(m1) << 23)));
}
// Byte c of w as 2^23 + byte: a permute, where a conversion has a quarter of its rate.
LUX_DEV float byte_bias(uint32_t w, int c) { return __uint_as_float(__byte_perm(w, 0x4b000000u, 0x7440 | c)); }
LUX_DEV float spatial_w(float f, int i) {  // SpatialW (:212-217)
  float d = fabsf(__fsub_rn(f, (float)(i * 2)));
  d = d < 1.0f ? d : 1.0f;
  return f2i(d) == 0 ? 1.0f : __uint_as_float(0x3eaaaaabu);
}

// BilateralUpsampleFromCollapse (:166-209) for one output pixel. inverse: lo = rcp(prev) and out = rcp(V/S) (the InverseDepth
// steps).
LUX_DEV float bilateral_pixel(const float* __restrict__ prev, int lw, int lh, const uint8_t* __restrict__ guide, int gstride,
                              const uint8_t* __restrict__ g2, float k, bool inverse, const uint32_t* __restrict__ rcp_table, int x, int y) {
  const float eps = __uint_as_float(0x322bcc77u);
  int wm1 = lw - 1, hm1 = lh - 1;
  int iy0 = (y - 1) / 2;
  float fy = __fadd_rn((float)y, -0.5f);
  const uint8_t* o = guide + ((size_t)y * gstride + x) * 4;
  float hr = o[0], hg = o[1], hb = o[2];
  int ix0 = (x - 1) / 2;
  float fx = __fadd_rn((float)x, -0.5f);
  int ibx = ix0 < 0 ? 0 : ix0;
  if (ibx > wm1) ibx = wm1;
  float wx0 = spatial_w(fx, ibx);
  int ix1 = ix0 + 1;
  if (ix1 < 0) ix1 = 0;
  if (ix1 > wm1) ix1 = wm1;
  float wx1 = spatial_w(fx, ix1);
  float accV = 0.0f, accS = 0.0f;
  for (int j = 0; j < 2; j++) {
    int iy = iy0 + j;
    if (iy < 0) iy = 0;
    if (iy > hm1) iy = hm1;
    float wy = spatial_w(fy, iy);
    size_t lrow = (size_t)iy * lw;
    const uint8_t* q = g2 + (lrow + ibx) * 4;
    float d0 = __fsub_rn(hr, (float)q[0]), d1 = __fsub_rn(hg, (float)q[1]), d2 = __fsub_rn(hb, (float)q[2]);
    float s = __fadd_rn(__fmul_rn(d1, d1), __fadd_rn(__fmul_rn(d2, d2), __fmul_rn(d0, d0)));
    float t = -__fmul_rn(s, k);
    float w0 = __fmul_rn(__fadd_rn(up_exp2(t), eps), __fmul_rn(wy, wx0));
    q = g2 + (lrow + ix1) * 4;
    d0 = __fsub_rn(hr, (float)q[0]); d1 = __fsub_rn(hg, (float)q[1]); d2 = __fsub_rn(hb, (float)q[2]);
    s = __fadd_rn(__fmul_rn(d1, d1), __fadd_rn(__fmul_rn(d2, d2), __fmul_rn(d0, d0)));
    t = -__fmul_rn(s, k);
    float w1 = __fmul_rn(__fadd_rn(up_exp2(t), eps), __fmul_rn(wy, wx1));
    float l0 = prev[lrow + ibx], l1 = prev[lrow + ix1];
    if (inverse) { l0 = rcp_approx(l0, rcp_table); l1 = rcp_approx(l1, rcp_table); }
    float v0 = __fmul_rn(l0, w0), v1 = __fmul_rn(l1, w1);
    accV = __fadd_rn(v1, __fadd_rn(v0, accV));
    accS = __fadd_rn(w1, __fadd_rn(w0, accS));
  }
  const float r = __fdiv_rn(accV, accS);
  return inverse ? rcp_approx(r, rcp_table) : r;
}

// What one upsample reads and writes: the depth and, where conf is not null, the confidence.
struct Bilateral {
  const float *prev, *conf;
  int lw, lh;
  const uint8_t* guide;
  int W, H, gstride;
  const uint8_t* g2;
  float k;
  const uint32_t* rcp;
  float *out, *out_conf;
  int qx, qy;  // quads: output pixels 1..2·qx by 1..2·qy
  uint64_t minus0;  // for mul_alone
};

// Every output pixel by itself, of the depth and the confidence or one of them: guides that are not word-aligned, and images
// too small for the quads.
template <bool DEPTH, bool CONF>
__global__ void __launch_bounds__(128) k_bilateral_pixels(const Bilateral b) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  if (x >= b.W) return;
  for (int y = blockIdx.y; y < b.H; y += gridDim.y) {  // gridDim.y is capped at 65535 rows; taller images loop
    const size_t at = (size_t)y * b.W + x;
    if (DEPTH) b.out[at] = bilateral_pixel(b.prev, b.lw, b.lh, b.guide, b.gstride, b.g2, b.k, true, b.rcp, x, y);
    if (CONF) b.out_conf[at] = bilateral_pixel(b.conf, b.lw, b.lh, b.guide, b.gstride, b.g2, b.k, false, b.rcp, x, y);
  }
}

// The output pixels outside the quads, one by one: row 0 and the rows past the quads, then column 0 and the columns past
// them.
__global__ void k_bilateral_border(const Bilateral b) {
  const int top = b.H - 2 * b.qy, side = b.W - 2 * b.qx;  // rows and columns outside the quads
  const size_t n = (size_t)top * b.W + (size_t)side * 2 * b.qy;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    int x, y;
    if (i < (size_t)top * b.W) {
      const int r = (int)(i / b.W);
      x = (int)(i - (size_t)r * b.W);
      y = r == 0 ? 0 : 2 * b.qy + r;
    } else {
      const size_t j = i - (size_t)top * b.W;
      const int r = (int)(j / side), c = (int)(j - (size_t)r * side);
      y = 1 + r;
      x = c == 0 ? 0 : 2 * b.qx + c;
    }
    b.out[(size_t)y * b.W + x] = bilateral_pixel(b.prev, b.lw, b.lh, b.guide, b.gstride, b.g2, b.k, true, b.rcp, x, y);
    if (b.conf) b.out_conf[(size_t)y * b.W + x] = bilateral_pixel(b.conf, b.lw, b.lh, b.guide, b.gstride, b.g2, b.k, false, b.rcp, x, y);
  }
}

// Output pixels 2i + 1 and 2i + 2 of rows 2j + 1 and 2j + 2 share their four low-resolution pixels (i, i + 1) x (j, j + 1): a
// thread makes the four, loading and inverting the low pixels once, and the confidence with the depth's weights. The
// spatial weights are then 1 for the nearer column or row and a third for the farther one. The two taps of a row run in one
// register pair. Persistent blocks, as many as are resident, with the rcpps table in shared memory. Bound by issue: depth and
// confidence of 4160x3120 88 us; scalar taps took 128, one thread an output pixel and a launch each 297.
constexpr int kQuadBlocks = 5;  // of 256 threads an SM, by their registers
template <bool CONF>
__global__ void __launch_bounds__(256, kQuadBlocks) k_bilateral_quads(const Bilateral b) {
  __shared__ uint32_t tab[4096];
  for (int i = threadIdx.x; i < 1024; i += 256) reinterpret_cast<uint4*>(tab)[i] = __ldg(reinterpret_cast<const uint4*>(b.rcp) + i);
  __syncthreads();
  auto rcp = [&](float v) {  // rcp_entry, as selections
    const uint32_t u = fbits(v), r = tab[(u >> 11) & 0xfff], sign = u & 0x80000000u, a = u & 0x7fffffffu;
    const int re = (int)((r >> 23) & 0xff) + 127 - (int)(a >> 23);
    uint32_t o = sign | (re > 0 ? (uint32_t)re << 23 | (r & 0x7fffffu) : 0u);
    o = a < 0x800000u ? sign | 0x7f800000u : o;
    return ffrom(a < 0x7f800000u ? o : a == 0x7f800000u ? sign : u | 0x400000u);
  };
  const float eps = __uint_as_float(0x322bcc77u), third = __uint_as_float(0x3eaaaaabu), third2 = __fmul_rn(third, third);
  const F2 near_far[2][2] = {{f2(1.0f, third), f2(third, 1.0f)}, {f2(third, third2), f2(third2, third)}};
  const unsigned n = (unsigned)b.qx * (unsigned)b.qy, step = gridDim.x * 256u;
  for (unsigned t = blockIdx.x * 256u + threadIdx.x; t < n; t += step) {
    const int j = (int)(t / (unsigned)b.qx), i = (int)(t - (unsigned)j * (unsigned)b.qx);
    F2 lo[2], cf[2], q[2][3];  // low pixels (0, r), (1, r); the guide's negated
    uint32_t hw[4];
#pragma unroll
    for (int o = 0; o < 4; o++)
      hw[o] = __ldg(reinterpret_cast<const uint32_t*>(b.guide) + (2 * (size_t)j + 1 + (o >> 1)) * b.gstride + 2 * i + 1 + (o & 1));
#pragma unroll
    for (int r = 0; r < 2; r++) {
      const size_t p = (size_t)(j + r) * b.lw + i;
      lo[r] = f2(rcp(__ldg(b.prev + p)), rcp(__ldg(b.prev + p + 1)));
      if (CONF) cf[r] = f2(__ldg(b.conf + p), __ldg(b.conf + p + 1));
      const uint32_t w0 = __ldg(reinterpret_cast<const uint32_t*>(b.g2) + p), w1 = __ldg(reinterpret_cast<const uint32_t*>(b.g2) + p + 1);
#pragma unroll
      for (int ch = 0; ch < 3; ch++) q[r][ch] = f2(-byte_bias(w0, ch), -byte_bias(w1, ch));
    }
#pragma unroll
    for (int o = 0; o < 4; o++) {  // the output pixel (o & 1, o >> 1) of the quad
      float accV = 0.0f, accS = 0.0f, accC = 0.0f;
#pragma unroll
      for (int r = 0; r < 2; r++) {
        F2 d[3];
#pragma unroll
        for (int ch = 0; ch < 3; ch++) {
          const float h = byte_bias(hw[o], ch);  // both sides of the difference carry the 2^23
          d[ch] = f2(h, h) + q[r][ch];
          d[ch] = d[ch] * d[ch];  // (whole numbers below 2^18 in all: no rounding)
        }
        float e0, e1, w0, w1, v0, v1;
        f2_get((d[1] + (d[2] + d[0])) * f2(b.k, b.k), e0, e1);
        const F2 wt = (up_exp2_neg(e0, e1, F2{b.minus0}) + f2(eps, eps)) * near_far[(o >> 1) != r][o & 1];
        f2_get(lo[r] * wt, v0, v1);
        accV = __fadd_rn(v1, __fadd_rn(v0, accV));
        if (CONF) {
          f2_get(cf[r] * wt, v0, v1);
          accC = __fadd_rn(v1, __fadd_rn(v0, accC));
        }
        f2_get(wt, w0, w1);
        accS = __fadd_rn(w1, __fadd_rn(w0, accS));
      }
      const size_t at = (2 * (size_t)j + 1 + (o >> 1)) * b.W + 2 * i + 1 + (o & 1);
      b.out[at] = rcp(__fdiv_rn(accV, accS));
      if (CONF) b.out_conf[at] = __fdiv_rn(accC, accS);
    }
  }
}

void launch_upsample(const float* prev, int pw, int ph, const uint8_t* guide, int gw, int gh, int gstride, float sigma,
                     const uint32_t* rcp_table, uint8_t* g2, float* out_depth, const float* prev_conf, float* out_conf,
                     cudaStream_t s) {
  double sy = (double)gh * 65536.0 / (double)ph, sx = (double)gw * 65536.0 / (double)pw;
  const int stepY = sy >= 2147483648.0 ? 0x7fffffff : (int)sy;
  const int stepX = sx >= 2147483648.0 ? 0x7fffffff : (int)sx;
  dim3 g1((pw + 127) / 128, std::min(ph, 65535));
  const bool words = (reinterpret_cast<uintptr_t>(guide) & 3) == 0;  // a caller's guide may lie at any address
  if (words) k_shift_resize<true><<<g1, 128, 0, s>>>(guide, gw, gh, gstride, pw, ph, stepX, stepY, g2);
  else k_shift_resize<false><<<g1, 128, 0, s>>>(guide, gw, gh, gstride, pw, ph, stepX, stepY, g2);
  volatile float ss = sigma * sigma;
  Bilateral b;
  b.prev = prev; b.lw = pw; b.lh = ph; b.guide = guide; b.W = gw; b.H = gh; b.gstride = gstride; b.g2 = g2;
  b.k = 0.5f / ss;
  b.rcp = rcp_table;
  b.out = out_depth;
  b.conf = prev_conf && out_conf ? prev_conf : nullptr;
  b.out_conf = out_conf;
  b.minus0 = 0x8000000080000000ull;
  // the quads whose four low pixels exist; their exponents are <= -0.0 for a positive finite k, float holds their coordinates
  // exactly below 2^23, and a 32-bit index counts them
  const bool quads = words && b.k > 0.0f && b.k <= 3.4e38f && gw < (1 << 23) && gh < (1 << 23) && (size_t)pw * ph < ((size_t)1 << 31);
  b.qx = quads ? std::max(0, std::min((gw - 1) / 2, pw - 1)) : 0;
  b.qy = quads ? std::max(0, std::min((gh - 1) / 2, ph - 1)) : 0;
  int launches = 2;
  // Below 150,000 quads, or 30,000 with confidence, the table's way into shared memory and the border's launch cost more than
  // they save (us a call, quads / pixels: 260x195 25 / 21, 400x300 27.1 / 26.4, 520x390 29 / 33; with confidence 130x98 25 / 24,
  // 200x150 25 / 25, 260x195 25 / 28).
  if ((size_t)b.qx * b.qy < (b.conf ? 30000 : 150000)) {
    const dim3 grid((gw + 127) / 128, std::min(gh, 65535));
    if (!b.conf) k_bilateral_pixels<true, false><<<grid, 128, 0, s>>>(b);
    else if (!words) k_bilateral_pixels<true, true><<<grid, 128, 0, s>>>(b);
    else {  // (three launches, as every aligned upsample with confidence)
      k_bilateral_pixels<true, false><<<grid, 128, 0, s>>>(b);
      k_bilateral_pixels<false, true><<<grid, 128, 0, s>>>(b);
      launches++;
    }
  } else {
    const unsigned grid = (unsigned)std::min<size_t>(((size_t)b.qx * b.qy + 255) / 256, 148 * kQuadBlocks);
    if (b.conf) k_bilateral_quads<true><<<grid, 256, 0, s>>>(b);
    else k_bilateral_quads<false><<<grid, 256, 0, s>>>(b);
    const size_t rest = (size_t)(gh - 2 * b.qy) * gw + (size_t)(gw - 2 * b.qx) * 2 * b.qy;  // row 0 at least
    k_bilateral_border<<<(unsigned)std::min<size_t>((rest + 127) / 128, 148 * 64), 128, 0, s>>>(b);
    launches++;
  }
  count_launches(launches);
}

}  // namespace lux
