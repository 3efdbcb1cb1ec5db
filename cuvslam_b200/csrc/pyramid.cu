// Fused pyramid + gradient kernel.
//
// One launch ("stage") takes an input level s that is already in memory (the uint8 frame for
// s = 0, else the FP32 level s) and produces up to NL further levels and their gradients.  Each CTA
// owns a T x T core tile of the deepest produced level and the matching 2^k-times larger core tiles
// of the shallower levels.  It stages the input region (with the halo the deeper levels and the
// 7-tap derivatives need) in shared memory, computes every intermediate level in shared memory,
// and writes each level's core image, grad_x and grad_y once, coalesced.  Level l+1 therefore never
// re-reads level l from HBM inside a stage.
//
// Arithmetic follows the reference exactly:
//   gaussian_scaling_kernel (image_pyramid.cu:56-102): 25 taps visited row-major, each as an FMA
//     into the accumulator, mirror addressing -x-1 / 2n-x-1, taps outside in both x and y skipped;
//   conv_grad_x/y_kernel (convolutions.cu:74-139): 7 taps j = -3..3 as FMAs, 0 within 3 px of
//     the border.
// so every level and gradient is bit-identical to the reference.
//
// Region geometry (1-D; the same in y).  With the deepest core [X, X+T) at level s+NL:
//   level s+NL is needed on [X-3, X+T+3)                (its own gradient halo), size S_NL = T+6;
//   level s+k  is needed on [2a-2, 2b+1) given [a, b) at level s+k+1, size S_k = 2 S_{k+1} + 3.
// Mirrored taps near the image border fall inside these regions (the region always reaches the
// border it is mirrored about), so a CTA never reads outside its shared-memory tiles.
#include <cuda_runtime.h>

#include "fe_common.cuh"
#include "fe_internal.h"

namespace fe {

namespace {

// Generic stages: the deepest level's core tile is KT x KT (8 or 16, chosen by the batch autotuner).
constexpr int kThreads = 256;

__host__ __device__ constexpr int region_size(int kt, int nl, int k) {
  return k == nl ? kt + 6 : 2 * region_size(kt, nl, k + 1) + 3;
}
__host__ __device__ constexpr int smem_floats(int kt, int nl) {
  int s = 0;
  for (int k = 0; k <= nl; ++k) s += region_size(kt, nl, k) * region_size(kt, nl, k);
  return s;
}

template <typename InT>
__device__ __forceinline__ float load_px(const InT* base, int64_t pitch_bytes, int x, int y) {
  const InT* row = reinterpret_cast<const InT*>(reinterpret_cast<const char*>(base) + (int64_t)y * pitch_bytes);
  return (float)__ldg(row + x);
}

// One output of gaussian_scaling_kernel at level coordinates (x, y), reading the source level from
// a shared-memory region whose origin is (ax, ay) and row length is `stride`.
__device__ __forceinline__ float downscale_px(const float* src, int stride, int ax, int ay, int sw, int sh, int x,
                                              int y) {
  const float k1[5] = {1.f / 16.f, 4.f / 16.f, 6.f / 16.f, 4.f / 16.f, 1.f / 16.f};
  const int x0 = 2 * x - 2, y0 = 2 * y - 2;
  float acc = 0.f;
  if (x0 >= 0 && y0 >= 0 && x0 + 4 < sw && y0 + 4 < sh) {
    const float* p = src + (y0 - ay) * stride + (x0 - ax);
#pragma unroll
    for (int k = 0; k < 5; ++k)
#pragma unroll
      for (int l = 0; l < 5; ++l) acc = __fmaf_rn(k1[k] * k1[l], p[k * stride + l], acc);
    return acc;
  }
  // the five columns and rows first, so that the 25 loads do not wait on one another (a skipped
  // corner tap's cell lies in the image too)
  int xi[5], yi[5];
  bool xo[5], yo[5];
#pragma unroll
  for (int l = 0; l < 5; ++l) {
    xo[l] = x0 + l < 0 || x0 + l >= sw;
    yo[l] = y0 + l < 0 || y0 + l >= sh;
    xi[l] = mirror_index(x0 + l, sw) - ax;
    yi[l] = (mirror_index(y0 + l, sh) - ay) * stride;
  }
#pragma unroll
  for (int k = 0; k < 5; ++k) {
#pragma unroll
    for (int l = 0; l < 5; ++l) {
      const float f = __fmaf_rn(k1[k] * k1[l], src[yi[k] + xi[l]], acc);
      acc = xo[l] && yo[k] ? acc : f;
    }
  }
  return acc;
}

// The two rings of cells around the w x h image that lie in a shared-memory region of rw x rh cells
// (row length `stride`) whose origin is (ax, ay): each takes the value the mirror addressing reads
// there (-x-1 / 2n-x-1), so that the decimation's taps need no index arithmetic near the edges.  A
// frame's time is that of its slowest tile where all tiles run at once: the mirrored path per pixel
// made a corner tile four times as long as an inner one (levels 1-2 of the FP32 stage 21 500 cycles,
// 4 700 with the cells in place).
template <int NT, typename T>
__device__ __forceinline__ void mirror_rings(T* buf, int stride, int rw, int rh, int ax, int ay, int w, int h,
                                             int tid) {
  for (int i = tid; i < 4 * (rw + rh); i += NT) {
    const bool col = i < 4 * rh;  // columns -2, -1, w, w + 1 over the rows, then the rows over the image's columns
    const int k = col ? i : i - 4 * rh;
    const int m = k & 3, p = k >> 2;
    const int x = col ? (m < 2 ? m - 2 : w + m - 2) : ax + p, y = col ? ay + p : (m < 2 ? m - 2 : h + m - 2);
    const int cx = x - ax, cy = y - ay;
    if (cx < 0 || cx >= rw || cy < 0 || cy >= rh || y < -2 || y > h + 1 || (!col && (x < 0 || x >= w))) continue;
    const int sx = mirror_index(x, w) - ax, sy = mirror_index(y, h) - ay;
    if (sx < 0 || sx >= rw || sy < 0 || sy >= rh) continue;
    buf[cy * stride + cx] = buf[sy * stride + sx];
  }
}

// 25-tap value at an interior place, or at one whose mirrored cells are in place: taps row by row.
__device__ __forceinline__ float downscale_25(const float* p, int stride) {
  const float k1[5] = {1.f / 16.f, 4.f / 16.f, 6.f / 16.f, 4.f / 16.f, 1.f / 16.f};
  float acc = 0.f;
#pragma unroll
  for (int k = 0; k < 5; ++k)
#pragma unroll
    for (int l = 0; l < 5; ++l) acc = __fmaf_rn(k1[k] * k1[l], p[k * stride + l], acc);
  return acc;
}

// Whether (x, y) is a corner pixel of a w x h level: the only pixels whose windows reach outside in x
// and in y, where gaussian_scaling_kernel leaves taps out.
__device__ __forceinline__ bool is_corner(int x, int y, int w, int h) {
  return (x == 0 || x == w - 1) && (y == 0 || y == h - 1);
}

// Levels tail[0..n) of one camera from the complete level `src` (global), by one CTA: the source
// level is copied to shared memory (L2, bypassing L1), each tail level's image is computed there
// with the 25-tap rule and its gradients from it.  `smem` holds kTailFloats floats.
__device__ void stage_tail(const Level& src, const Level* tail, int n, float* smem) {
  float* a = smem;                              // current source level (w x h, row stride w)
  int sw = src.w, sh = src.h;
  for (int i = threadIdx.x; i < sw * sh; i += kThreads) {
    const int r = i / sw, c = i - r * sw;
    cp_async4(a + i, src.img + (size_t)r * src.pitch + c);
  }
  cp_async_wait_all();
  __syncthreads();
  for (int t = 0; t < n; ++t) {
    const Level& L = tail[t];
    float* b = a + sw * sh;                     // this level, right after its source
    for (int i = threadIdx.x; i < L.w * L.h; i += kThreads) {
      const int y = i / L.w, x = i - y * L.w;
      const float v = downscale_px(a, sw, 0, 0, sw, sh, x, y);
      b[i] = v;
      L.img[(size_t)y * L.pitch + x] = v;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < L.w * L.h; i += kThreads) {
      const int y = i / L.w, x = i - y * L.w;
      const float* p = b + i;
      float gx = 0.f, gy = 0.f;
      if (x > 2 && x < L.w - 3) {
#pragma unroll
        for (int j = 0; j < 7; ++j)
          if (j != 3) gx = __fmaf_rn(dsp_tap(j), p[j - 3], gx);
      }
      if (y > 2 && y < L.h - 3) {
#pragma unroll
        for (int j = 0; j < 7; ++j)
          if (j != 3) gy = __fmaf_rn(dsp_tap(j), p[(j - 3) * L.w], gy);
      }
      L.gx[(size_t)y * L.pitch + x] = gx;
      if (L.gy) L.gy[(size_t)y * L.pitch + x] = gy;
    }
    __syncthreads();
    // the next level's source: move this level to the front (it is smaller than its source)
    for (int i = threadIdx.x; i < L.w * L.h; i += kThreads) a[i] = b[i];  // disjoint ranges
    __syncthreads();
    sw = L.w;
    sh = L.h;
  }
}

// (five blocks per SM: the straight-line edge path takes 54 registers unbounded, with which four blocks fit and a
// two-level build of a 4096x4096 uint8 frame takes 461 us; 407 us at 48 registers, 418 with the edges in a loop)
template <typename InT, int NL, int KT>
__global__ void __launch_bounds__(kThreads, 5) pyramid_stage_kernel(const __grid_constant__ StageBatch batch) {
  extern __shared__ float smem[];
  // camera of this CTA: last job whose tile_begin <= blockIdx.x
  int lo = 0, hi = batch.njobs - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (batch.job[mid].tile_begin <= (int)blockIdx.x) lo = mid; else hi = mid - 1;
  }
  const StageJob& job = batch.job[lo];
  const int t = (int)blockIdx.x - job.tile_begin;
  const int X = (t % job.tiles_x) * KT, Y = (t / job.tiles_x) * KT;

  int a[NL + 1], S[NL + 1], off[NL + 1];
  a[NL] = X - 3;
  int ay[NL + 1];
  ay[NL] = Y - 3;
#pragma unroll
  for (int k = NL - 1; k >= 0; --k) {
    a[k] = 2 * a[k + 1] - 2;
    ay[k] = 2 * ay[k + 1] - 2;
  }
  int o = 0;
#pragma unroll
  for (int k = 0; k <= NL; ++k) {
    S[k] = region_size(KT, NL, k);
    off[k] = o;
    o += S[k] * S[k];
  }

  // 1. stage the input region (FP32 sources as asynchronous copies, all in flight at once), scaled
  //    by job.scale (the first stage of a scaled build; 1 otherwise)
  {
    const int w = job.src_w, h = job.src_h;
    const InT* src = static_cast<const InT*>(job.src);
    float* dst = smem + off[0];
    for (int i = threadIdx.x; i < S[0] * S[0]; i += kThreads) {
      const int r = i / S[0], c = i - r * S[0];
      const int gx = a[0] + c, gy = ay[0] + r;
      const bool in = gx >= 0 && gy >= 0 && gx < w && gy < h;
      if constexpr (sizeof(InT) == 4) {
        if (in) {
          cp_async4(dst + i, reinterpret_cast<const float*>(reinterpret_cast<const char*>(src) +
                                                            (int64_t)gy * job.src_pitch_bytes) + gx);
        } else {
          dst[i] = 0.f;
        }
      } else {
        dst[i] = in ? load_px(src, job.src_pitch_bytes, gx, gy) : 0.f;
      }
    }
    if constexpr (sizeof(InT) == 4) cp_async_wait_all();
    __syncthreads();
    if (job.scale != 1.f) {
      for (int i = threadIdx.x; i < S[0] * S[0]; i += kThreads) dst[i] = __fmul_rn(dst[i], job.scale);
      __syncthreads();
    }
  }

  // 2. deeper levels inside shared memory
#pragma unroll
  for (int k = 1; k <= NL; ++k) {
    const int sw = job.out[k - 1].w, sh = job.out[k - 1].h;
    const int w = job.out[k].w, h = job.out[k].h;
    const float* src = smem + off[k - 1];
    float* dst = smem + off[k];
    for (int i = threadIdx.x; i < S[k] * S[k]; i += kThreads) {
      const int r = i / S[k], c = i - r * S[k];
      const int gx = a[k] + c, gy = ay[k] + r;
      if (gx >= 0 && gy >= 0 && gx < w && gy < h)
        dst[i] = downscale_px(src, S[k - 1], a[k - 1], ay[k - 1], sw, sh, gx, gy);
    }
    __syncthreads();
  }

  // 3. core outputs: image, grad_x, grad_y
#pragma unroll
  for (int k = (job.write_level0 ? 0 : 1); k <= NL; ++k) {
    const Level& L = job.out[k];
    const int C = KT << (NL - k);
    const int cx0 = X << (NL - k), cy0 = Y << (NL - k);
    const float* reg = smem + off[k];
    for (int i = threadIdx.x; i < C * C; i += kThreads) {
      const int r = i / C, c = i - r * C;
      const int x = cx0 + c, y = cy0 + r;
      if (x >= L.w || y >= L.h) continue;
      const float* p = reg + (y - ay[k]) * S[k] + (x - a[k]);
      float sx = 0.f, sy = 0.f;
      if (x > 2 && x < L.w - 3) {
#pragma unroll
        for (int j = 0; j < 7; ++j)
          if (j != 3) sx = __fmaf_rn(dsp_tap(j), p[j - 3], sx);
      }
      if (y > 2 && y < L.h - 3) {
#pragma unroll
        for (int j = 0; j < 7; ++j)
          if (j != 3) sy = __fmaf_rn(dsp_tap(j), p[(j - 3) * S[k]], sy);
      }
      const int64_t o2 = (int64_t)y * L.pitch + x;
      L.img[o2] = p[0];
      L.gx[o2] = sx;
      if (L.gy) L.gy[o2] = sy;
    }
  }

  // 4. tail: the last CTA of the job computes the remaining (small) levels from the complete
  //    deepest level, in shared memory (threadfence + counter: every CTA's stores precede its count)
  if (job.tail_levels > 0) {
    __shared__ int last;
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence();
      last = atomicAdd(job.done, 1) == job.tiles_x * job.tiles_y - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    stage_tail(job.out[NL], job.tail, job.tail_levels, smem);
    if (threadIdx.x == 0) *job.done = 0;
  }
}

// ---------------------------------------------------------------- levels 0-2 from the uint8 frame
//
// The first stage dominates the pyramid's HBM traffic (it writes ~98% of the bytes), so it has its
// own kernel.  A CTA owns a 32x32 level-2 core tile (128x128 at level 0) and
//   1. stages its 176x163 uint8 tile with one TMA copy (zero fill outside the frame), or with plain
//      loads when the frame's base/pitch are not 16-byte aligned, and applies the optional box
//      prefilter to it (integer arithmetic, exact);
//   2. computes level 1 on its 79x79 region as column strips with a sliding 5-row window of
//      horizontal 5-tap sums, in integers;
//   3. computes level 2 on its 38x38 region the same way from level 1, in FP32;
//   4. writes the three core tiles (image, grad_x, grad_y) with 16-byte stores.
// Levels 1 and 2 are exact in any summation order (all partial sums are multiples of 2^-16 below
// 2^8), so the separable sums equal gaussian_scaling_kernel's 25-tap FMA chain bit for bit; only the
// four image-corner pixels, where the reference skips the taps outside in both x and y, are redone
// with the 25-tap rule.
namespace l012 {

// Level-1 and level-2 regions of a T2 x T2 level-2 core tile, in x and y: level 1 [2X2-8, 2X2+2T2+7),
// level 2 rows [Y2-3, Y2+T2+3), columns stored from X2-4.
template <int T2>
struct Geo {
  static constexpr int kThreads = 16 * T2;
  static constexpr int kS1 = 2 * T2 + 15, kS1S = 2 * T2 + 16;
  static constexpr int kS2 = T2 + 6, kS2S = T2 + 8;
};

constexpr int kT2 = 32;
constexpr int kThreads = Geo<kT2>::kThreads;
constexpr int kS0W = 176, kS0H = 163;  // uint8 tile: cols [4X2-32, 4X2+144), rows [4Y2-19, 4Y2+144)
constexpr int kS1 = Geo<kT2>::kS1, kS1S = Geo<kT2>::kS1S;
constexpr int kS2 = Geo<kT2>::kS2, kS2S = Geo<kT2>::kS2S;
constexpr int kB0Bytes = kS0W * kS0H;
constexpr int kOffB1 = (kB0Bytes + 127) / 128 * 128;
constexpr int kOffB2 = kOffB1 + kS1 * kS1S * 4;
constexpr int kOffBar = kOffB2 + kS2 * kS2S * 4;
constexpr int kSmem = kOffBar + 64;
// with the box prefilter: the prefiltered tile after the rest
constexpr int kOffBox = (kSmem + 127) / 128 * 128;
constexpr int kSmemBox = kOffBox + kB0Bytes;

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

// Bounded wait on an mbarrier phase: false when `limit` polls all found it incomplete (the caller
// reports it and gives up).
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t phase, int limit) {
  for (int i = 0; i < limit; ++i) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(smem_u32(bar)), "r"(phase)
        : "memory");
    if (done) return true;
  }
  return false;
}

// Bytes k and k+1 of a word as exact floats: 0x4B0000bb is 2^23 + b, then subtract 2^23.
__device__ __forceinline__ float2 bytes_to_float2(uint32_t wd, int k) {
  const float lo = __uint_as_float(__byte_perm(wd, 0x4B000000u, 0x7540u + k));
  const float hi = __uint_as_float(__byte_perm(wd, 0x4B000000u, 0x7540u + k + 1));
  return __fadd2_rn(make_float2(lo, hi), make_float2(-8388608.f, -8388608.f));
}

// 25-tap value with the reference's corner rule (taps outside in x and y skipped), uint8 source.
__device__ float corner_l1(const uint8_t* B0, int a0x, int a0y, int w0, int h0, int x1, int y1) {
  int acc = 0, xi[5], yi[5];
  bool xo[5], yo[5];
#pragma unroll
  for (int l = 0; l < 5; ++l) {
    const int xc = 2 * x1 - 2 + l, yc = 2 * y1 - 2 + l;
    xo[l] = xc < 0 || xc >= w0;
    yo[l] = yc < 0 || yc >= h0;
    xi[l] = mirror_index(xc, w0) - a0x;
    yi[l] = (mirror_index(yc, h0) - a0y) * kS0W;
  }
#pragma unroll
  for (int k = 0; k < 5; ++k)
#pragma unroll
    for (int l = 0; l < 5; ++l) {
      const int wk = k == 2 ? 6 : (k & 1 ? 4 : 1), wl = l == 2 ? 6 : (l & 1 ? 4 : 1);
      const int v = wk * wl * (int)B0[yi[k] + xi[l]];
      acc += xo[l] && yo[k] ? 0 : v;
    }
  return (float)acc * (1.f / 256.f);
}

// Deeper levels (3 and below) inside the same launch.  Every tile CTA also writes its 16x16 core of
// level 3's image (its sources lie in the tile's level-2 region).  The launch's CTAs take work items
// from an atomic queue: each camera's tiles, then (placed after the next camera's tiles, so that
// their inputs are usually complete when they are taken) its deeper-level items:
//   band items of phase d (d = level 3, then level 4 when needed): level d's gradients and level
//     d+1's image for a band of rows, from level d's rows staged in shared memory;
//   one rest item: the remaining levels from the first one that fits in shared memory, staged once,
//     each further level computed there.
// An item waits (bounded) until the items it reads from are counted complete: tiles for phase 3,
// phase-3 bands for phase 4, the last banded phase (or the tiles) for the rest.  Items are taken in
// queue order and only wait on earlier items, which are running or done, so the waits end.  Pixels
// follow the reference's rules (25-tap decimation with mirror and corner skip, 7-tap derivatives),
// so every level is bit-identical to the reference's.
constexpr int kDeepFloats = (kOffBar / 4) & ~3;

// The block's thread count NT is a template parameter of the deeper-level code.
// Rows [lo, lo + rows) of level L into sm (row stride `stride` floats, a multiple of 4), through L2.
template <int NT>
__device__ __forceinline__ void stage_rows(const Level& L, int lo, int rows, int stride, float* sm) {
  const int q4 = L.w >> 2, rem = L.w & 3;
  for (int i = threadIdx.x; i < rows * q4; i += NT) {
    const int r = i / q4, c = (i - r * q4) * 4;
    const float* g = L.img + (size_t)(lo + r) * L.pitch + c;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(sm + r * stride + c)), "l"(g) : "memory");
  }
  if (rem)
    for (int i = threadIdx.x; i < rows * rem; i += NT) {
      const int r = i / rem, c = (q4 << 2) + (i - r * rem);
      sm[r * stride + c] = __ldcg(L.img + (size_t)(lo + r) * L.pitch + c);
    }
  cp_async_wait_all();
  __syncthreads();
}

// Gradients of rows [y0, y1) of level D whose image rows [lo, ...) are in sm (row stride `stride`, a
// multiple of 4; 16-byte aligned): four pixels per work item, the taps as 16-byte loads.
template <int NT>
__device__ __forceinline__ void smem_gradients(const Level& D, const float* a, int stride, int lo, int y0, int y1) {
  const int w = D.w, h = D.h, q4 = (w + 3) >> 2;
  for (int i = threadIdx.x; i < (y1 - y0) * q4; i += NT) {
    const int r = i / q4, y = y0 + r, x = (i - r * q4) * 4;
    const float* p = a + (y - lo) * stride + x;
    const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 lq = x >= 4 ? *reinterpret_cast<const float4*>(p - 4) : z;
    const float4 mq = *reinterpret_cast<const float4*>(p);
    const float4 rq = x + 4 < stride ? *reinterpret_cast<const float4*>(p + 4) : z;
    const float v[12] = {lq.x, lq.y, lq.z, lq.w, mq.x, mq.y, mq.z, mq.w, rq.x, rq.y, rq.z, rq.w};
    float gx[4] = {0.f, 0.f, 0.f, 0.f}, gy[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      float g = 0.f;
#pragma unroll
      for (int j = 0; j < 7; ++j)
        if (j != 3) g = __fmaf_rn(dsp_tap(j), v[1 + k + j], g);
      gx[k] = x + k > 2 && x + k < w - 3 ? g : 0.f;
    }
    if (y > 2 && y < h - 3) {
#pragma unroll
      for (int j = 0; j < 7; ++j) {
        if (j == 3) continue;
        const float4 c = *reinterpret_cast<const float4*>(p + (j - 3) * stride);
        gy[0] = __fmaf_rn(dsp_tap(j), c.x, gy[0]);
        gy[1] = __fmaf_rn(dsp_tap(j), c.y, gy[1]);
        gy[2] = __fmaf_rn(dsp_tap(j), c.z, gy[2]);
        gy[3] = __fmaf_rn(dsp_tap(j), c.w, gy[3]);
      }
    }
    const size_t o = (size_t)y * D.pitch + x;
    if (x + 3 < w) {
      *reinterpret_cast<float4*>(D.gx + o) = make_float4(gx[0], gx[1], gx[2], gx[3]);
      if (D.gy) *reinterpret_cast<float4*>(D.gy + o) = make_float4(gy[0], gy[1], gy[2], gy[3]);
    } else {
      for (int k = 0; k < 4 && x + k < w; ++k) {
        D.gx[o + k] = gx[k];
        if (D.gy) D.gy[o + k] = gy[k];
      }
    }
  }
}

// Band item: level S's gradients on rows [2 r0, 2 r1) and level N's image on rows [r0, r1).
template <int NT>
__device__ void band_item(const Level& S, const Level& N, int r0, int nrows, float* sm) {
  const int r1 = min(N.h, r0 + nrows);
  const int ss = (S.w + 3) & ~3;
  const int lo = max(0, 2 * r0 - 3), hi = min(S.h - 1, 2 * r1 + 2);
  stage_rows<NT>(S, lo, hi - lo + 1, ss, sm);
  smem_gradients<NT>(S, sm, ss, lo, min(S.h, 2 * r0), min(S.h, 2 * r1));
  for (int i = threadIdx.x; i < (r1 - r0) * N.w; i += NT) {
    const int y = r0 + i / N.w, x = i - (i / N.w) * N.w;
    N.img[(size_t)y * N.pitch + x] = downscale_px(sm, ss, 0, lo, S.w, S.h, x, y);
  }
}

// Rest item: levels tail[0..n): tail[0]'s image is complete; its gradients and every further level.
template <int NT>
__device__ void rest_item(const Level* tail, int n, float* sm) {
  const int s0 = (tail[0].w + 3) & ~3;
  stage_rows<NT>(tail[0], 0, tail[0].h, s0, sm);
  const float* a = sm;
  int as = s0;
  float* b = sm + s0 * tail[0].h;
  for (int t = 0; t < n; ++t) {
    const Level& D = tail[t];
    if (t > 0) {
      const Level& S = tail[t - 1];
      const int ds = (D.w + 3) & ~3;
      for (int i = threadIdx.x; i < D.w * D.h; i += NT) {
        const int y = i / D.w, x = i - y * D.w;
        const float v = downscale_px(a, as, 0, 0, S.w, S.h, x, y);
        b[y * ds + x] = v;
        D.img[(size_t)y * D.pitch + x] = v;
      }
      __syncthreads();
      a = b;
      as = ds;
      b += ds * D.h;
    }
    smem_gradients<NT>(D, a, as, 0, 0, D.h);
  }
}

// Thread 0 waits (at most batch.wait_limit polls) until *ctr >= target; false (and status bit 1)
// when the wait ran out.
template <typename Batch>
__device__ bool wait_count(const Batch& batch, int* ctr, int target) {
  __shared__ int s_ok;
  if (threadIdx.x == 0) {
    int ok = 0;
    for (int i = 0; i < batch.wait_limit; ++i) {
      if (*reinterpret_cast<volatile int*>(ctr) >= target) {
        ok = 1;
        break;
      }
      __nanosleep(64);
    }
    if (!ok && batch.status) atomicOr(batch.status, 2);
    __threadfence();
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

// Deeper-level item idx of job J.  J.done: [0] tiles finished, [1] phase-3 bands, [2] phase-4
// bands; the launch's last CTA returns them to zero for the next launch (not the rest item: if one
// of its waits gave up, tiles and bands may still be counting).
template <int NT, typename Batch>
__device__ void deep_item(const Batch& batch, const StageJob& J, int idx, float* sm) {
  int* ctr = J.done;
  const int ntiles = J.tiles_x * J.tiles_y;
  const int nb0 = J.deep_bands[0], nb1 = J.deep_bands[1];
  if (idx < nb0 + nb1) {
    const int ph = idx < nb0 ? 0 : 1, b = ph ? idx - nb0 : idx;
    if (wait_count(batch, ph ? ctr + 1 : ctr, ph ? nb0 : ntiles))
      band_item<NT>(J.tail[ph], J.tail[ph + 1], b * J.deep_band_rows[ph], J.deep_band_rows[ph], sm);
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence();
      atomicAdd(ctr + 1 + ph, 1);
    }
  } else {
    const int r = J.deep_rest;
    if (wait_count(batch, r == 0 ? ctr : ctr + r, r == 0 ? ntiles : J.deep_bands[r - 1]))
      rest_item<NT>(J.tail + r, J.tail_levels - r, sm);
  }
}

// The box prefilter of the reference (CudaBoxPrefilter::prefilter, box_prefilter.cpp:31-38: a
// [1 2 1]/4 pass along x, then along y truncated to an integer, then the frame's one-pixel border ring
// copied from the input) on the staged uint8 tile: on integer input every partial sum is exact, so
// an interior pixel is (sum of [1 2 1] x [1 2 1] weighted bytes) >> 4.  Four columns per thread
// item, as packed 16-bit lanes (sums stay below 2^12); rows 1..kS0H-2 and every column are written
// (the tile's outermost rows and columns, never read, keep their input bytes).  Pixels on the
// frame's border ring take the input byte.
__device__ void box3_tile(const uint8_t* raw, uint8_t* out, int a0x, int a0y, int w0, int h0) {
  constexpr int kWords = kS0W / 4;            // four-column groups per row
  constexpr int kBand = 15;                   // rows per thread item
  constexpr int kBands = (kS0H - 2 + kBand - 1) / kBand;
  const uint32_t* rw = reinterpret_cast<const uint32_t*>(raw);
  for (int it = threadIdx.x; it < kWords * kBands; it += kThreads) {
    const int c4 = it % kWords, band = it / kWords;
    const int r0 = 1 + band * kBand, r1 = min(kS0H - 1, r0 + kBand);
    // horizontal [1 2 1] of four columns as two words of 16-bit lanes (columns c, c+1 | c+2, c+3)
    auto hsum = [&](int r, uint32_t& lo, uint32_t& hi) {
      const uint32_t w = rw[r * kWords + c4];
      const uint32_t wl = c4 > 0 ? rw[r * kWords + c4 - 1] : 0u;
      const uint32_t wr = c4 + 1 < kWords ? rw[r * kWords + c4 + 1] : 0u;
      // zero-extended byte pairs (selector nibbles 4-7 pick the second operand; masks clear the rest)
      const uint32_t cl = __byte_perm(w, 0u, 0x4140), ch = __byte_perm(w, 0u, 0x4342);  // c, c+1 | c+2, c+3
      const uint32_t mid = __byte_perm(w, 0u, 0x4241);                                   // c+1, c+2
      const uint32_t left = __byte_perm(wl, w, 0x4443) & 0x00ff00ffu;                    // c-1, c
      const uint32_t right = __byte_perm(w, wr, 0x4443) & 0x00ff00ffu;                   // c+3, c+4
      lo = left + 2u * cl + mid;
      hi = mid + 2u * ch + right;
    };
    uint32_t a_lo, a_hi, b_lo, b_hi, c_lo, c_hi;
    hsum(r0 - 1, a_lo, a_hi);
    hsum(r0, b_lo, b_hi);
    for (int r = r0; r < r1; ++r) {
      hsum(r + 1, c_lo, c_hi);
      const uint32_t vlo = ((a_lo + 2u * b_lo + c_lo) >> 4) & 0x0fff0fffu;
      const uint32_t vhi = ((a_hi + 2u * b_hi + c_hi) >> 4) & 0x0fff0fffu;
      reinterpret_cast<uint32_t*>(out)[r * kWords + c4] = __byte_perm(vlo, vhi, 0x6420);
      a_lo = b_lo; a_hi = b_hi;
      b_lo = c_lo; b_hi = c_hi;
    }
  }
  // rows 0 and kS0H-1 of the tile: input bytes
  for (int i = threadIdx.x; i < 2 * kS0W; i += kThreads) {
    const int r = i < kS0W ? 0 : kS0H - 1, c = i < kS0W ? i : i - kS0W;
    out[r * kS0W + c] = raw[r * kS0W + c];
  }
  __syncthreads();
  // the frame's border ring: input bytes (rows 0 and h0-1, columns 0 and w0-1 inside the tile)
  for (int i = threadIdx.x; i < 2 * (kS0W + kS0H); i += kThreads) {
    int r, c;
    if (i < 2 * kS0W) {
      r = (i < kS0W ? 0 : h0 - 1) - a0y;
      c = i % kS0W;
    } else {
      const int k = i - 2 * kS0W;
      c = (k < kS0H ? 0 : w0 - 1) - a0x;
      r = k % kS0H;
    }
    if (r >= 0 && r < kS0H && c >= 0 && c < kS0W) out[r * kS0W + c] = raw[r * kS0W + c];
  }
}

// Image and gradients of the tile's level-1 and level-2 cores from their shared-memory regions (no grad_y
// where a level has no such plane: a current or secondary pyramid may come without them).
template <int T2>
__device__ __forceinline__ void levels12_outputs(const Level& L1, const Level& L2, const float* B1, const float* B2,
                                                 int X2, int Y2, int tid) {
  using G = Geo<T2>;
  constexpr int kQ1 = 2 * T2 * (T2 / 2), kQ2 = T2 * (T2 / 4);  // four-pixel items of levels 1 and 2
#pragma unroll 1
  for (int q = tid; q < kQ1 + kQ2; q += G::kThreads) {
    const bool lev1 = q < kQ1;
    const int qq = lev1 ? q : q - kQ1;
    const Level& L = lev1 ? L1 : L2;
    const int qpr = lev1 ? T2 / 2 : T2 / 4;
    const int y = (lev1 ? 2 * Y2 : Y2) + qq / qpr, x = (lev1 ? 2 * X2 : X2) + (qq % qpr) * 4;
    if (y >= L.h || x >= L.w) continue;
    const float* T = lev1 ? B1 : B2;
    const int stride = lev1 ? G::kS1S : G::kS2S;
    const int r = y - (lev1 ? 2 * Y2 - 8 : Y2 - 3), c = x - (lev1 ? 2 * X2 - 8 : X2 - 4);
    float v[12];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const float4 f = *reinterpret_cast<const float4*>(T + r * stride + c - 4 + 4 * k);
      v[4 * k] = f.x;
      v[4 * k + 1] = f.y;
      v[4 * k + 2] = f.z;
      v[4 * k + 3] = f.w;
    }
    // pixel pairs (x, x+1), (x+2, x+3): packed FP32x2 FMA chains, vertical taps as 16-byte loads
    float2 sx[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
    float2 sy[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
    for (int j = 0; j < 7; ++j) {
      if (j == 3) continue;
      const float2 d = make_float2(dsp_tap(j), dsp_tap(j));
      const float4 cv = *reinterpret_cast<const float4*>(T + (r - 3 + j) * stride + c);
      sx[0] = __ffma2_rn(d, make_float2(v[1 + j], v[2 + j]), sx[0]);
      sx[1] = __ffma2_rn(d, make_float2(v[3 + j], v[4 + j]), sx[1]);
      sy[0] = __ffma2_rn(d, make_float2(cv.x, cv.y), sy[0]);
      sy[1] = __ffma2_rn(d, make_float2(cv.z, cv.w), sy[1]);
    }
    float gx[4] = {sx[0].x, sx[0].y, sx[1].x, sx[1].y};
    float gy[4] = {sy[0].x, sy[0].y, sy[1].x, sy[1].y};
    const bool vin = y > 2 && y < L.h - 3;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (!(x + i > 2 && x + i < L.w - 3)) gx[i] = 0.f;
      if (!vin) gy[i] = 0.f;
    }
    const int64_t o = (int64_t)y * L.pitch + x;
    if (x + 3 < L.w) {
      *reinterpret_cast<float4*>(L.img + o) = make_float4(v[4], v[5], v[6], v[7]);
      *reinterpret_cast<float4*>(L.gx + o) = make_float4(gx[0], gx[1], gx[2], gx[3]);
      if (L.gy) *reinterpret_cast<float4*>(L.gy + o) = make_float4(gy[0], gy[1], gy[2], gy[3]);
    } else {
      for (int i = 0; i < 4 && x + i < L.w; ++i) {
        L.img[o + i] = v[4 + i];
        L.gx[o + i] = gx[i];
        if (L.gy) L.gy[o + i] = gy[i];
      }
    }
  }
}

// Tile t of job: levels 0-2, and when the launch computes the deeper levels, level 3's image core
// (after which the tile counts itself complete in job.done[0]).
template <typename Batch>
__device__ __forceinline__ void l012_tile(const Batch& batch, const StageJob& job, int t, unsigned char* sm) {
  uint8_t* B0 = sm;
  float* B1 = reinterpret_cast<float*>(sm + kOffB1);
  float* B2 = reinterpret_cast<float*>(sm + kOffB2);
  uint64_t* bar = reinterpret_cast<uint64_t*>(sm + kOffBar);
  const int tid = threadIdx.x;
  const int X2 = (t % job.tiles_x) * kT2, Y2 = (t / job.tiles_x) * kT2;
  const Level& L0 = job.out[0];
  const Level& L1 = job.out[1];
  const Level& L2 = job.out[2];
  const int w0 = L0.w, h0 = L0.h, w1 = L1.w, h1 = L1.h, w2 = L2.w, h2 = L2.h;
  const int a0x = 4 * X2 - 32, a0y = 4 * Y2 - 19;
  const int a1x = 2 * X2 - 8, a1y = 2 * Y2 - 8;
  const int a2x = X2 - 4, a2y = Y2 - 3;  // level-2 storage origin (column X2-4 is never computed)

  // 1. the uint8 tile
  if (job.use_tma) {
    if (tid == 0) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(bar)));
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (tid == 0) {
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(kB0Bytes)
                   : "memory");
      asm volatile(
          "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], "
          "[%4];" ::"r"(smem_u32(B0)),
          "l"(reinterpret_cast<uint64_t>(&job.tmap)), "r"(a0x), "r"(a0y), "r"(smem_u32(bar))
          : "memory");
    }
    const bool ok = mbar_wait(bar, 0, batch.wait_limit);
    if (__syncthreads_or(!ok)) {
      if (tid == 0 && batch.status) atomicOr(batch.status, 1);
      // the copy may still land: wait once more, with the full bound whatever the launch's limit, so
      // no write targets a retired CTA
      mbar_wait(bar, 0, kDefaultWaitLimit);
      if (job.tail_levels > 0 && tid == 0) atomicAdd(job.done, 1);  // still counted (its level 3 is not written)
      return;
    }
  } else {
    // four columns per item: the two aligned words around them shifted into place where both lie inside
    // the frame's bytes, single bytes (zero outside the frame) elsewhere
    const uint8_t* src = static_cast<const uint8_t*>(job.src);
    const uint8_t* last = src + (int64_t)(h0 - 1) * job.src_pitch_bytes + w0;
    uint32_t* dst = reinterpret_cast<uint32_t*>(B0);
#pragma unroll 4
    for (int i = tid; i < kS0H * (kS0W / 4); i += kThreads) {
      const int r = i / (kS0W / 4), gx = a0x + (i - r * (kS0W / 4)) * 4, gy = a0y + r;
      uint32_t v = 0;
      if (gy >= 0 && gy < h0 && gx > -4 && gx < w0) {
        const uint8_t* q = src + (int64_t)gy * job.src_pitch_bytes + gx;
        const uint8_t* al = reinterpret_cast<const uint8_t*>(reinterpret_cast<uintptr_t>(q) & ~(uintptr_t)3);
        if (gx >= 0 && gx + 3 < w0 && al >= src && al + 8 <= last) {
          const uint32_t lo = __ldg(reinterpret_cast<const uint32_t*>(al));
          const uint32_t hi = __ldg(reinterpret_cast<const uint32_t*>(al + 4));
          v = __funnelshift_r(lo, hi, 8 * (uint32_t)(q - al));
        } else {
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if (gx + k >= 0 && gx + k < w0) v |= (uint32_t)__ldg(q + k) << (8 * k);
        }
      }
      dst[i] = v;
    }
  }
  __syncthreads();
  if (job.box3) {
    uint8_t* F = sm + kOffBox;
    box3_tile(B0, F, a0x, a0y, w0, h0);
    B0 = F;
    __syncthreads();
  }

  // tiles at the frame's edges: the mirrored cells each level's decimation reads are put in place, and
  // the image's corner pixels redone with the rule that leaves taps out
  const bool edge = a0x < 0 || a0y < 0 || a0x + kS0W > w0 || a0y + kS0H > h0;
  if (edge) {
    mirror_rings<kThreads>(B0, kS0W, kS0W, kS0H, a0x, a0y, w0, h0, tid);
    __syncthreads();
  }

  // 2. level 1 (integer sums: exact in any order): a thread takes a pair of columns (c, c + 1) and a
  //    band of 7 rows, sliding the 5-row window of horizontal sums down the band.  The taps of both
  //    columns are bytes 4 pp + 14 .. 4 pp + 20 of a staged row: three words, one byte permute and two
  //    dp4a with the weights (1, 4, 6, 4) plus the fifth tap.  Columns outside the image get values
  //    that nothing reads before mirror_rings replaces them.
  constexpr int kP1 = kS1S / 2, kB1 = 7;
  static_assert(kP1 * ((kS1 + kB1 - 1) / kB1) <= kThreads, "one item per thread");
  if (tid < kP1 * ((kS1 + kB1 - 1) / kB1)) {
    const int pp = tid % kP1, band = tid / kP1;
    const int c = 2 * pp;
    const int ys = max(a1y + band * kB1, 0), ye = min(a1y + min(band * kB1 + kB1, kS1), h1);
    if (ys < ye) {
      const bool two = c + 1 < kS1;  // the region's last column has no second one
      const uint8_t* p = B0 + (2 * ys - 2 - a0y) * kS0W + 4 * pp + 12;
      auto H2 = [&](const uint8_t* q, int& ha, int& hb) {
        const uint32_t wa = *reinterpret_cast<const uint32_t*>(q);
        const uint32_t wb = *reinterpret_cast<const uint32_t*>(q + 4);
        const uint32_t wc = two ? *reinterpret_cast<const uint32_t*>(q + 8) : 0u;
        ha = (int)__dp4a(__byte_perm(wa, wb, 0x5432u), 0x04060401u, (wb >> 16) & 0xffu);
        hb = (int)__dp4a(wb, 0x04060401u, wc & 0xffu);
      };
      int a0_, b0_, a1_, b1_, a2_, b2_, a3_, b3_, a4_, b4_;
      H2(p, a0_, b0_);
      H2(p + kS0W, a1_, b1_);
      H2(p + 2 * kS0W, a2_, b2_);
      p += 3 * kS0W;
      for (int y = ys;;) {
        H2(p, a3_, b3_);
        H2(p + kS0W, a4_, b4_);
        const int Sa = a0_ + a4_ + 4 * (a1_ + a3_) + 6 * a2_;
        const int Sb = b0_ + b4_ + 4 * (b1_ + b3_) + 6 * b2_;
        *reinterpret_cast<float2*>(B1 + (y - a1y) * kS1S + c) =
            make_float2((float)Sa * (1.f / 256.f), (float)Sb * (1.f / 256.f));
        if (++y >= ye) break;
        a0_ = a2_;
        b0_ = b2_;
        a1_ = a3_;
        b1_ = b3_;
        a2_ = a4_;
        b2_ = b4_;
        p += 2 * kS0W;
      }
    }
  }
  __syncthreads();
  if (edge && tid < 4) {
    const int x1 = (tid & 1) ? w1 - 1 : 0, y1 = (tid & 2) ? h1 - 1 : 0;
    if (x1 >= a1x && x1 < a1x + kS1 && y1 >= a1y && y1 < a1y + kS1)
      B1[(y1 - a1y) * kS1S + (x1 - a1x)] = corner_l1(B0, a0x, a0y, w0, h0, x1, y1);
  }
  if (edge) {
    __syncthreads();
    mirror_rings<kThreads>(B1, kS1S, kS1, kS1, a1x, a1y, w1, h1, tid);
    __syncthreads();
  }

  // 3. level 2 from level 1, same scheme in FP32 (exact: level 1 holds multiples of 1/256 below 256
  //    and every partial sum fits FP32's 24 bits): a pair of columns and a band of 3 rows per thread;
  //    both columns' taps are the level-1 values 4 pp .. 4 pp + 6 of a row (two 16-byte loads)
  constexpr int kP2 = kS2 / 2, kB2 = 3;
  if (tid < kP2 * ((kS2 + kB2 - 1) / kB2)) {
    const int pp = tid % kP2, band = tid / kP2;
    const int c = 2 * pp;
    const int x2 = X2 - 3 + c;
    const int ys = max(a2y + band * kB2, 0), ye = min(a2y + min(band * kB2 + kB2, kS2), h2);
    if (ys < ye) {
      const float* p = B1 + (2 * ys - 2 - a1y) * kS1S + 4 * pp;
      auto H2 = [&](const float* q, float& ha, float& hb) {
        const float4 u = *reinterpret_cast<const float4*>(q);
        const float4 v = *reinterpret_cast<const float4*>(q + 4);
        ha = (u.x + v.x) + 4.f * (u.y + u.w) + 6.f * u.z;
        hb = (u.z + v.z) + 4.f * (u.w + v.y) + 6.f * v.x;
      };
      float a0_, b0_, a1_, b1_, a2_, b2_, a3_, b3_, a4_, b4_;
      H2(p, a0_, b0_);
      H2(p + kS1S, a1_, b1_);
      H2(p + 2 * kS1S, a2_, b2_);
      p += 3 * kS1S;
      for (int y = ys;;) {
        H2(p, a3_, b3_);
        H2(p + kS1S, a4_, b4_);
        float* o = B2 + (y - a2y) * kS2S + (x2 - a2x);
        o[0] = ((a0_ + a4_) + 4.f * (a1_ + a3_) + 6.f * a2_) * (1.f / 256.f);
        o[1] = ((b0_ + b4_) + 4.f * (b1_ + b3_) + 6.f * b2_) * (1.f / 256.f);
        if (++y >= ye) break;
        a0_ = a2_;
        b0_ = b2_;
        a1_ = a3_;
        b1_ = b3_;
        a2_ = a4_;
        b2_ = b4_;
        p += 2 * kS1S;
      }
    }
  }
  __syncthreads();
  if (edge) {
    if (tid < 4) {
      const int x2 = (tid & 1) ? w2 - 1 : 0, y2 = (tid & 2) ? h2 - 1 : 0;
      if (x2 >= X2 - 3 && x2 < X2 + kT2 + 3 && y2 >= a2y && y2 < a2y + kS2)
        B2[(y2 - a2y) * kS2S + (x2 - a2x)] = downscale_px(B1, kS1S, a1x, a1y, w1, h1, x2, y2);
    }
    __syncthreads();
    mirror_rings<kThreads>(B2, kS2S, kS2S, kS2, a2x, a2y, w2, h2, tid);
    __syncthreads();
  }
  // level 3's image on this tile's core (its sources [X2-2, X2+T2+2) lie in the level-2 region), when
  // the launch computes the deeper levels
  if (job.tail_levels > 0) {
    constexpr int kT3 = kT2 / 2;
    if (tid < kT3 * kT3) {
      const Level& L3 = job.tail[0];
      const int x3 = (X2 >> 1) + (tid % kT3), y3 = (Y2 >> 1) + (tid / kT3);
      if (x3 < L3.w && y3 < L3.h)
        L3.img[(size_t)y3 * L3.pitch + x3] =
            is_corner(x3, y3, L3.w, L3.h) ? downscale_px(B2, kS2S, a2x, a2y, w2, h2, x3, y3)
                                          : downscale_25(B2 + (2 * y3 - 2 - a2y) * kS2S + (2 * x3 - 2 - a2x), kS2S);
    }
    // the deeper-level items read only level 3's image: count the tile now, while its level 0-2
    // stores (issued below) are not yet outstanding, so the fence has only these writes to wait for
    __syncthreads();
    if (tid == 0) {
      __threadfence();
      atomicAdd(job.done, 1);
    }
  }

  // 4. core outputs
  // level 0 from the uint8 tile.  Bytes become floats exactly as (2^23 + b) - 2^23 (a byte
  // permute into the mantissa, then one packed subtract per pair); the 7-tap derivatives of pixel
  // pairs run as packed FP32x2 FMAs, each lane rounding exactly as the scalar FMA chain.
  // (a) image and grad_y: a thread takes a pixel pair's column over a strip of 16 rows and slides the
  //     derivative's 7-row window down it in registers, so each byte is converted once per strip.
  {
    constexpr int kRows = kT2 / 2;
    const int pc = tid % (2 * kT2), strip = tid / (2 * kT2);  // 64 pairs x 8 strips of 16 rows
    const int x = 4 * X2 + 2 * pc, y0 = 4 * Y2 + kRows * strip;
    if (x < w0 && y0 < h0) {
      const uint8_t* colp = B0 + (y0 - a0y - 3) * kS0W + (x - a0x);  // rows y0-3 .. y0+kRows+2
      auto pair = [&](int k) {
        return bytes_to_float2((uint32_t)*reinterpret_cast<const uint16_t*>(colp + k * kS0W), 0);
      };
      const bool two = x + 1 < w0;
      float2 win[7];
#pragma unroll
      for (int k = 0; k < 6; ++k) win[k] = pair(k);
#pragma unroll
      for (int i = 0; i < kRows; ++i) {
        win[6] = pair(i + 6);
        const int y = y0 + i;
        if (y < h0) {
          float2 gy = make_float2(0.f, 0.f);
#pragma unroll
          for (int j = 0; j < 7; ++j) {
            if (j == 3) continue;
            gy = __ffma2_rn(make_float2(dsp_tap(j), dsp_tap(j)), win[j], gy);
          }
          if (!(y > 2 && y < h0 - 3)) gy = make_float2(0.f, 0.f);
          const int64_t o = (int64_t)y * L0.pitch + x;
          if (two) {
            *reinterpret_cast<float2*>(L0.img + o) = win[3];
            *reinterpret_cast<float2*>(L0.gy + o) = gy;
          } else {
            L0.img[o] = win[3].x;
            L0.gy[o] = gy.x;
          }
        }
#pragma unroll
        for (int k = 0; k < 6; ++k) win[k] = win[k + 1];
      }
    }
  }
  // (b) grad_x: a thread takes four pixels of a row and their horizontal neighbours x-4 .. x+7.
#pragma unroll 1
  for (int q = tid; q < 4 * kT2 * kT2; q += kThreads) {
    const int y = 4 * Y2 + q / kT2, x = 4 * X2 + (q % kT2) * 4;
    if (y >= h0 || x >= w0) continue;
    const uint8_t* p = B0 + (y - a0y) * kS0W + (x - a0x);
    const uint32_t wl = *reinterpret_cast<const uint32_t*>(p - 4);
    const uint32_t wm = *reinterpret_cast<const uint32_t*>(p);
    const uint32_t wr = *reinterpret_cast<const uint32_t*>(p + 4);
    const float2 v[6] = {bytes_to_float2(wl, 0), bytes_to_float2(wl, 2), bytes_to_float2(wm, 0),
                         bytes_to_float2(wm, 2), bytes_to_float2(wr, 0), bytes_to_float2(wr, 2)};
    // pixel x+i needs v at flat indices 1+i+j (j = 0..6); pairs (i, i+1) for i = 0, 2
    auto hv = [&](int f) { return (f & 1) ? make_float2(v[f >> 1].y, v[(f >> 1) + 1].x) : v[f >> 1]; };
    float2 gx2[2];
#pragma unroll
    for (int pp = 0; pp < 2; ++pp) {
      float2 sx = make_float2(0.f, 0.f);
#pragma unroll
      for (int j = 0; j < 7; ++j) {
        if (j == 3) continue;
        sx = __ffma2_rn(make_float2(dsp_tap(j), dsp_tap(j)), hv(1 + 2 * pp + j), sx);
      }
      gx2[pp] = sx;
    }
    float gx[4] = {gx2[0].x, gx2[0].y, gx2[1].x, gx2[1].y};
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (!(x + i > 2 && x + i < w0 - 3)) gx[i] = 0.f;
    const int64_t o = (int64_t)y * L0.pitch + x;
    if (x + 3 < w0) {
      *reinterpret_cast<float4*>(L0.gx + o) = make_float4(gx[0], gx[1], gx[2], gx[3]);
    } else {
      for (int i = 0; i < 4 && x + i < w0; ++i) L0.gx[o + i] = gx[i];
    }
  }
  levels12_outputs<kT2>(L1, L2, B1, B2, X2, Y2, tid);
}

// MINB: CTAs resident per SM the registers are budgeted for (2, or 3 with fewer registers).
template <int MINB, typename Batch>
__global__ void __launch_bounds__(kThreads, MINB) pyramid_l012_kernel(const __grid_constant__ Batch batch) {
  extern __shared__ __align__(128) unsigned char sm[];
  __shared__ int s_q;
  const int tid = threadIdx.x;
  if (tid == 0) s_q = batch.queue ? atomicAdd(batch.queue, 1) : (int)blockIdx.x;
  __syncthreads();
  const int q = s_q;
  int j = 0, idx = 0;
  bool deep = false;
  for (; j < batch.njobs; ++j) {
    const StageJob& J = batch.job[j];
    if (q >= J.tile_begin && q < J.tile_begin + J.tiles_x * J.tiles_y) {
      idx = q - J.tile_begin;
      break;
    }
    if (J.tail_levels > 0 && q >= J.q_deep && q < J.q_deep + J.deep_items) {
      idx = q - J.q_deep;
      deep = true;
      break;
    }
  }
  if (j < batch.njobs) {
    const StageJob& job = batch.job[j];
    if (!deep) {
      l012_tile(batch, job, idx, sm);
    } else {
      deep_item<kThreads>(batch, job, idx, reinterpret_cast<float*>(sm));
    }
  }
  if (batch.queue) {
    // the last CTA to finish returns the queue and the jobs' item counters to zero for the next
    // launch: every other CTA has counted itself finished after its own counter updates
    __syncthreads();
    if (tid == 0) {
      __threadfence();
      if (atomicAdd(batch.queue + 1, 1) == (int)gridDim.x - 1) {
        __threadfence();
        for (int k = 0; k < batch.njobs; ++k)
          if (batch.job[k].tail_levels > 0) {
            batch.job[k].done[0] = 0;
            batch.job[k].done[1] = 0;
            batch.job[k].done[2] = 0;
          }
        batch.queue[0] = 0;
        batch.queue[1] = 0;
      }
    }
  }
}

}  // namespace l012

// ---------------------------------------------------------------- levels 0-2 from an FP32 frame
//
// The first stage of an FP32 build (FP32 frames, the level 0 of an RGB frame, the adjoint's planes):
// a CTA owns a 16x16 level-2 core tile (64x64 at level 0), stages its 100x97 FP32 region with one TMA
// copy (plain asynchronous copies when the frame's base or pitch are not 16-byte aligned), computes
// the level-1 and level-2 regions in shared memory and writes the three cores and level 3's image
// core.  FP32 sums are not exact, so every output keeps gaussian_scaling_kernel's 25-tap row-major
// FMA chain: a thread takes a pair of columns and a strip of rows, loads each source row's seven
// values once and adds them into every output of the strip that they are a tap of (an output still
// sees its taps row by row).  Bound by shared memory and issue, not by HBM: sixteen 1280x720 frames take
// 76 us here plus 9 us for the deeper levels (352 us with the generic stages' one pixel per thread), one
// 1921x1201 frame 13 + 12 us (85 us).
namespace lead {

constexpr int kT2 = 16;
using G = l012::Geo<kT2>;
constexpr int kThreads = G::kThreads;
constexpr int kW = 4 * kT2 + 36, kH = 4 * kT2 + 33;  // level 0: cols [4X2-20, 4X2+80), rows [4Y2-18, 4Y2+79)
constexpr int kOffB1 = (kW * kH * 4 + 127) / 128 * 128;
constexpr int kOffB2 = kOffB1 + G::kS1 * G::kS1S * 4;
constexpr int kOffBar = kOffB2 + G::kS2 * G::kS2S * 4;
constexpr int kSmem = kOffBar + 64;

// ROWS outputs of a column pair; load(k, v) gives the seven source values under both columns of the
// k-th source row of the strip.
template <int ROWS, typename Load>
__device__ __forceinline__ void down_pair(Load load, float2 (&acc)[ROWS]) {
  constexpr float k1[5] = {1.f / 16.f, 4.f / 16.f, 6.f / 16.f, 4.f / 16.f, 1.f / 16.f};
#pragma unroll
  for (int o = 0; o < ROWS; ++o) acc[o] = make_float2(0.f, 0.f);
#pragma unroll
  for (int k = 0; k < 2 * ROWS + 3; ++k) {
    float v[7];
    load(k, v);
#pragma unroll
    for (int o = 0; o < ROWS; ++o) {
      const int j = k - 2 * o;
      if (j < 0 || j > 4) continue;
#pragma unroll
      for (int l = 0; l < 5; ++l) {
        acc[o].x = __fmaf_rn(k1[j] * k1[l], v[l], acc[o].x);
        acc[o].y = __fmaf_rn(k1[j] * k1[l], v[l + 2], acc[o].y);
      }
    }
  }
}

template <typename Batch>
__global__ void __launch_bounds__(kThreads, 4) pyramid_lead_kernel(const __grid_constant__ Batch batch) {
  extern __shared__ __align__(128) unsigned char sm[];
  constexpr int kS1 = G::kS1, kS1S = G::kS1S, kS2 = G::kS2, kS2S = G::kS2S;
  float* B0 = reinterpret_cast<float*>(sm);
  float* B1 = reinterpret_cast<float*>(sm + kOffB1);
  float* B2 = reinterpret_cast<float*>(sm + kOffB2);
  uint64_t* bar = reinterpret_cast<uint64_t*>(sm + kOffBar);
  const int tid = threadIdx.x;
  int lo = 0, hi = batch.njobs - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (batch.job[mid].tile_begin <= (int)blockIdx.x) lo = mid; else hi = mid - 1;
  }
  const StageJob& job = batch.job[lo];
  const int t = (int)blockIdx.x - job.tile_begin;
  const int X2 = (t % job.tiles_x) * kT2, Y2 = (t / job.tiles_x) * kT2;
  const Level& L0 = job.out[0];
  const Level& L1 = job.out[1];
  const Level& L2 = job.out[2];
  const int w0 = L0.w, h0 = L0.h, w1 = L1.w, h1 = L1.h, w2 = L2.w, h2 = L2.h;
  const int a0x = 4 * X2 - 20, a0y = 4 * Y2 - 18;
  const int a1x = 2 * X2 - 8, a1y = 2 * Y2 - 8;
  const int a2x = X2 - 4, a2y = Y2 - 3;

  // 1. the FP32 region (X2 is a multiple of 16: the copy starts at a column multiple of 4), zero
  //    outside the frame, times job.scale
  if (job.use_tma) {
    if (tid == 0) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(l012::smem_u32(bar)));
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (tid == 0) {
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(l012::smem_u32(bar)),
                   "r"(kW * kH * 4)
                   : "memory");
      asm volatile(
          "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], "
          "[%4];" ::"r"(l012::smem_u32(B0)),
          "l"(reinterpret_cast<uint64_t>(&job.tmap)), "r"(a0x), "r"(a0y), "r"(l012::smem_u32(bar))
          : "memory");
    }
    if (__syncthreads_or(!l012::mbar_wait(bar, 0, batch.wait_limit))) {
      if (tid == 0 && batch.status) atomicOr(batch.status, 1);
      // the copy may still land: wait once more with the full bound, so that no write targets a
      // retired CTA
      l012::mbar_wait(bar, 0, kDefaultWaitLimit);
      return;
    }
  } else {
    const char* src = static_cast<const char*>(job.src);
    for (int i = tid; i < kW * kH; i += kThreads) {
      const int r = i / kW, c = i - r * kW;
      const int x = a0x + c, y = a0y + r;
      if (x >= 0 && y >= 0 && x < w0 && y < h0)
        cp_async4(B0 + i, reinterpret_cast<const float*>(src + (int64_t)y * job.src_pitch_bytes) + x);
      else
        B0[i] = 0.f;
    }
    cp_async_wait_all();
  }
  __syncthreads();
  if (job.scale != 1.f) {
    static_assert(kW * kH % 4 == 0, "whole float4s");
    float4* b = reinterpret_cast<float4*>(B0);
    for (int i = tid; i < kW * kH / 4; i += kThreads) {
      float4 v = b[i];
      v.x = __fmul_rn(v.x, job.scale);
      v.y = __fmul_rn(v.y, job.scale);
      v.z = __fmul_rn(v.z, job.scale);
      v.w = __fmul_rn(v.w, job.scale);
      b[i] = v;
    }
    __syncthreads();
  }
  // tiles at the frame's edges: the mirrored cells each level's decimation reads are put in place, and
  // the image's corner pixels redone with the rule that leaves taps out
  const bool edge = a0x < 0 || a0y < 0 || a0x + kW > w0 || a0y + kH > h0;
  if (edge) {
    mirror_rings<kThreads>(B0, kW, kW, kH, a0x, a0y, w0, h0, tid);
    __syncthreads();
  }

  // 2. level 1: 24 column pairs x 10 strips of 5 rows (the last strip overlaps the one before); both
  //    columns' taps are the staged columns 4 pp + 2 .. 4 pp + 8.  Cells outside the image get values
  //    that nothing reads before mirror_rings replaces them.
  {
    constexpr int kRows = 5, kP = kS1S / 2, kStrips = (kS1 + kRows - 1) / kRows;
    static_assert(kP * kStrips <= kThreads, "one strip per thread");
    if (tid < kP * kStrips) {
      const int pp = tid % kP, r = min((tid / kP) * kRows, kS1 - kRows), c = 2 * pp;
      const float* p = B0 + 2 * r * kW + 4 * pp + 2;
      const bool seven = c + 1 < kS1;  // the region's last column has no second one
      float2 acc[kRows];
      down_pair<kRows>(
          [&](int k, float* v) {
            const float* q = p + k * kW;
            const float2 a = *reinterpret_cast<const float2*>(q);
            const float4 b = *reinterpret_cast<const float4*>(q + 2);
            v[0] = a.x;
            v[1] = a.y;
            v[2] = b.x;
            v[3] = b.y;
            v[4] = b.z;
            v[5] = b.w;
            v[6] = seven ? q[6] : 0.f;
          },
          acc);
#pragma unroll
      for (int o = 0; o < kRows; ++o) *reinterpret_cast<float2*>(B1 + (r + o) * kS1S + c) = acc[o];
    }
  }
  __syncthreads();
  if (edge) {
    if (tid < 4) {
      const int x1 = (tid & 1) ? w1 - 1 : 0, y1 = (tid & 2) ? h1 - 1 : 0;
      if (x1 >= a1x && x1 < a1x + kS1 && y1 >= a1y && y1 < a1y + kS1)
        B1[(y1 - a1y) * kS1S + (x1 - a1x)] = downscale_px(B0, kW, a0x, a0y, w0, h0, x1, y1);
    }
    __syncthreads();
    mirror_rings<kThreads>(B1, kS1S, kS1, kS1, a1x, a1y, w1, h1, tid);
    __syncthreads();
  }

  // 3. level 2 from level 1: a column pair of one row per thread (source columns 4 pp .. 4 pp + 6)
  {
    constexpr int kP = kS2 / 2;
    static_assert(kP * kS2 <= kThreads, "one pair per thread");
    if (tid < kP * kS2) {
      const int pp = tid % kP, r = tid / kP, c = 2 * pp;
      const float* p = B1 + 2 * r * kS1S + 4 * pp;
      float2 acc[1];
      down_pair<1>(
          [&](int k, float* v) {
            const float4 a = *reinterpret_cast<const float4*>(p + k * kS1S);
            const float4 b = *reinterpret_cast<const float4*>(p + k * kS1S + 4);
            v[0] = a.x;
            v[1] = a.y;
            v[2] = a.z;
            v[3] = a.w;
            v[4] = b.x;
            v[5] = b.y;
            v[6] = b.z;
          },
          acc);
      float* o = B2 + r * kS2S + c + 1;  // columns are stored from X2 - 4
      o[0] = acc[0].x;
      o[1] = acc[0].y;
    }
  }
  __syncthreads();
  if (edge) {
    if (tid < 4) {
      const int x2 = (tid & 1) ? w2 - 1 : 0, y2 = (tid & 2) ? h2 - 1 : 0;
      if (x2 > a2x && x2 <= a2x + kS2 && y2 >= a2y && y2 < a2y + kS2)
        B2[(y2 - a2y) * kS2S + (x2 - a2x)] = downscale_px(B1, kS1S, a1x, a1y, w1, h1, x2, y2);
    }
    __syncthreads();
    mirror_rings<kThreads>(B2, kS2S, kS2S, kS2, a2x, a2y, w2, h2, tid);
    __syncthreads();
  }

  // 4. level 3's image core, when the job has deeper levels (pyramid_deep_kernel does the rest)
  if (job.tail_levels > 0 && tid < kT2 * kT2 / 4) {
    constexpr int kT3 = kT2 / 2;
    const Level& L3 = job.tail[0];
    const int x3 = (X2 >> 1) + tid % kT3, y3 = (Y2 >> 1) + tid / kT3;
    if (x3 < L3.w && y3 < L3.h)
      L3.img[(size_t)y3 * L3.pitch + x3] =
          is_corner(x3, y3, L3.w, L3.h) ? downscale_px(B2, kS2S, a2x, a2y, w2, h2, x3, y3)
                                        : downscale_25(B2 + (2 * y3 - 2 - a2y) * kS2S + (2 * x3 - 2 - a2x), kS2S);
  }

  // 5. level 0's core: a thread takes four columns of a strip of four rows, the derivative's 7-row
  //    window sliding down it in registers; packed FP32x2 FMA chains, each lane rounding as the scalar
  //    chain
  {
    constexpr int kRows = 4;
    static_assert(kT2 * (4 * kT2 / kRows) == kThreads, "one strip per thread");
    const int x = 4 * X2 + 4 * (tid % kT2), y0 = 4 * Y2 + kRows * (tid / kT2);
    if (x < w0 && y0 < h0) {
      const float* p = B0 + (y0 - a0y) * kW + (x - a0x);
      const bool img = !job.keep_level0;
      float4 win[7];
#pragma unroll
      for (int k = 0; k < 6; ++k) win[k] = *reinterpret_cast<const float4*>(p + (k - 3) * kW);
#pragma unroll
      for (int i = 0; i < kRows; ++i) {
        win[6] = *reinterpret_cast<const float4*>(p + (i + 3) * kW);
        const int y = y0 + i;
        if (y < h0) {
          const float4 l = *reinterpret_cast<const float4*>(p + i * kW - 4);
          const float4 r = *reinterpret_cast<const float4*>(p + i * kW + 4);
          const float v[12] = {l.x, l.y, l.z, l.w, win[3].x, win[3].y, win[3].z, win[3].w, r.x, r.y, r.z, r.w};
          float2 sx[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
          float2 sy[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
          for (int j = 0; j < 7; ++j) {
            if (j == 3) continue;
            const float2 d = make_float2(dsp_tap(j), dsp_tap(j));
            sx[0] = __ffma2_rn(d, make_float2(v[1 + j], v[2 + j]), sx[0]);
            sx[1] = __ffma2_rn(d, make_float2(v[3 + j], v[4 + j]), sx[1]);
            sy[0] = __ffma2_rn(d, make_float2(win[j].x, win[j].y), sy[0]);
            sy[1] = __ffma2_rn(d, make_float2(win[j].z, win[j].w), sy[1]);
          }
          float gx[4] = {sx[0].x, sx[0].y, sx[1].x, sx[1].y};
          float gy[4] = {sy[0].x, sy[0].y, sy[1].x, sy[1].y};
          const bool vin = y > 2 && y < h0 - 3;
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            if (!(x + k > 2 && x + k < w0 - 3)) gx[k] = 0.f;
            if (!vin) gy[k] = 0.f;
          }
          const int64_t o = (int64_t)y * L0.pitch + x;
          if (x + 3 < w0) {
            if (img) *reinterpret_cast<float4*>(L0.img + o) = win[3];
            *reinterpret_cast<float4*>(L0.gx + o) = make_float4(gx[0], gx[1], gx[2], gx[3]);
            if (L0.gy) *reinterpret_cast<float4*>(L0.gy + o) = make_float4(gy[0], gy[1], gy[2], gy[3]);
          } else {
            for (int k = 0; k < 4 && x + k < w0; ++k) {
              if (img) L0.img[o + k] = v[4 + k];
              L0.gx[o + k] = gx[k];
              if (L0.gy) L0.gy[o + k] = gy[k];
            }
          }
        }
#pragma unroll
        for (int k = 0; k < 6; ++k) win[k] = win[k + 1];
      }
    }
  }
  l012::levels12_outputs<kT2>(L1, L2, B1, B2, X2, Y2, tid);
}

// Levels 3 and below after pyramid_lead_kernel (level 3's image is complete): a cluster of eight CTAs
// per job, each level's rows split into eight bands: a band's gradients and the next level's image
// from its rows staged in shared memory (l012::band_item); a cluster barrier between levels.  The
// levels are read back through L2 (cp.async.cg, __ldcg), where the other CTAs' stores are.
constexpr int kDeepCtas = 8, kDeepThreads = 512, kDeepFloats = 12 * 1024;

template <typename Batch>
__global__ void __cluster_dims__(kDeepCtas, 1, 1) __launch_bounds__(kDeepThreads)
    pyramid_deep_kernel(const __grid_constant__ Batch batch) {
  extern __shared__ __align__(16) float dsm[];
  const StageJob& J = batch.job[blockIdx.x / kDeepCtas];
  const int rank = blockIdx.x % kDeepCtas;
  for (int t = 0; t < J.tail_levels; ++t) {
    const Level& S = J.tail[t];
    const int ss = (S.w + 3) & ~3;
    if (t + 1 < J.tail_levels) {
      const Level& N = J.tail[t + 1];
      const int per = (N.h + kDeepCtas - 1) / kDeepCtas, end = min(N.h, (rank + 1) * per);
      const int step = min(per, (kDeepFloats / ss - 6) / 2);
      for (int r0 = rank * per; r0 < end; r0 += step) {
        l012::band_item<kDeepThreads>(S, N, r0, min(step, end - r0), dsm);
        __syncthreads();
      }
      __threadfence();
      asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    } else {
      const int per = (S.h + kDeepCtas - 1) / kDeepCtas, end = min(S.h, (rank + 1) * per);
      const int step = min(per, kDeepFloats / ss - 6);
      for (int y0 = rank * per; y0 < end; y0 += step) {
        const int y1 = min(y0 + step, end), lo = max(0, y0 - 3);
        l012::stage_rows<kDeepThreads>(S, lo, min(S.h, y1 + 3) - lo, ss, dsm);
        l012::smem_gradients<kDeepThreads>(S, dsm, ss, lo, y0, y1);
        __syncthreads();
      }
    }
  }
}

}  // namespace lead

constexpr size_t stage_smem(int kt, int nl, bool tail = true) {
  return sizeof(float) * (tail && kTailFloats > smem_floats(kt, nl) ? kTailFloats : smem_floats(kt, nl));
}

template <typename InT, int NL, int KT>
cudaError_t set_stage_attr() {
  return cudaFuncSetAttribute(pyramid_stage_kernel<InT, NL, KT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)stage_smem(KT, NL));
}

template <typename InT, int NL>
cudaError_t launch_stage(const StageBatch& b, int tiles, int kt, bool tail, cudaStream_t s) {
  if ((kt & 31) == 16)
    pyramid_stage_kernel<InT, NL, 16><<<tiles, kThreads, stage_smem(16, NL, tail), s>>>(b);
  else
    pyramid_stage_kernel<InT, NL, 8><<<tiles, kThreads, stage_smem(8, NL, tail), s>>>(b);
  return cudaGetLastError();
}

template <int KT>
cudaError_t set_stage_attrs() {
  cudaError_t e;
  if ((e = set_stage_attr<uint8_t, 0, KT>()) != cudaSuccess) return e;
  if ((e = set_stage_attr<uint8_t, 1, KT>()) != cudaSuccess) return e;
  if ((e = set_stage_attr<uint8_t, 2, KT>()) != cudaSuccess) return e;
  if ((e = set_stage_attr<float, 0, KT>()) != cudaSuccess) return e;
  if ((e = set_stage_attr<float, 1, KT>()) != cudaSuccess) return e;
  return set_stage_attr<float, 2, KT>();
}

// ---------------------------------------------------------------- input stage
// Level 0 from an RGB8 frame, or from a small mono frame with the box prefilter (larger mono frames
// get the prefilter inside the levels 0-2 kernel).

// box_blur_x, then box_blur_y (convolutions.cu:141-205): [1 2 1]/4 along x, then along y, truncated.
__device__ __forceinline__ float box_h(float l, float c, float r) {
  return __fmaf_rn(0.25f, r, __fmaf_rn(0.5f, c, __fmul_rn(0.25f, l)));
}
__device__ __forceinline__ float box_v(float a, float b, float c) {
  const float t = __fmaf_rn(0.25f, c, __fmaf_rn(0.5f, b, __fmul_rn(0.25f, a)));
  return (float)(__float2uint_rz(t) & 0xffu);
}

// Small mono frame with the prefilter: one thread per pixel.
__global__ void input_mono_kernel(const uint8_t* src, int64_t pitch, int box3, int w, int h, float* dst, int64_t dp) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
  if (x >= w || y >= h) return;
  const uint8_t* p = src + (int64_t)y * pitch + x;
  float v = (float)p[0];
  if (box3 && x > 0 && x < w - 1 && y > 0 && y < h - 1) {
    float col[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const uint8_t* q = p + (int64_t)(k - 1) * pitch;
      col[k] = box_h((float)q[-1], (float)q[0], (float)q[1]);
    }
    v = box_v(col[0], col[1], col[2]);
  }
  dst[(int64_t)y * dp + x] = v;
}

// RGB frame: a thread takes four pixels of four rows; each row's 18 bytes (pixels x - 1 .. x + 4) come as
// six aligned words shifted into place, single bytes near the frame's ends; the prefilter's horizontal
// sums slide down the rows.  (A thread per pixel that read its nine neighbours' 27 bytes one by one took
// 18.9 us for 1921x1201 with the prefilter, this 8.4 us.)
constexpr int kRgbRows = 4;

__global__ void __launch_bounds__(256) input_rgb_kernel(const uint8_t* src, int64_t pitch, int box3, int w, int h,
                                                        float* dst, int64_t dp) {
  const int x = (blockIdx.x * 32 + (threadIdx.x & 31)) * 4, y0 = (blockIdx.y * 8 + (threadIdx.x >> 5)) * kRgbRows;
  if (x >= w || y0 >= h) return;
  const uint8_t* end = src + (int64_t)(h - 1) * pitch + 3 * (int64_t)w;
  // gray of pixels x - 1 .. x + 4 of row y (pixels outside the frame: any value)
  auto gray6 = [&](int y, float (&g)[6]) {
    const uint8_t* p = src + (int64_t)y * pitch + 3 * (int64_t)(x - 1);
    const uint8_t* al = reinterpret_cast<const uint8_t*>(reinterpret_cast<uintptr_t>(p) & ~(uintptr_t)3);
    uint32_t b[5];
    if (al >= src && al + 24 <= end) {
      uint32_t wd[6];
#pragma unroll
      for (int k = 0; k < 6; ++k) wd[k] = __ldg(reinterpret_cast<const uint32_t*>(al) + k);
      const uint32_t sh = 8 * (uint32_t)(p - al);
#pragma unroll
      for (int k = 0; k < 5; ++k) b[k] = __funnelshift_r(wd[k], wd[k + 1], sh);
    } else {
#pragma unroll
      for (int k = 0; k < 5; ++k) b[k] = 0;
#pragma unroll
      for (int k = 0; k < 18; ++k)
        if (x - 1 + k / 3 >= 0 && x - 1 + k / 3 < w) b[k >> 2] |= (uint32_t)__ldg(p + k) << (8 * (k & 3));
    }
    auto byte = [&](int k) { return (float)((b[k >> 2] >> (8 * (k & 3))) & 0xffu); };
#pragma unroll
    for (int i = 0; i < 6; ++i)
      // the expression of cast_image_kernel_rgb (image_cast.cu:60-66) as nvcc contracts it
      g[i] = __fmaf_rn(0.114f, byte(3 * i + 2), __fmaf_rn(0.299f, byte(3 * i), __fmul_rn(0.587f, byte(3 * i + 1))));
  };
  auto put = [&](int y, const float (&v)[4]) {
    float* o = dst + (int64_t)y * dp + x;
    if (x + 3 < w) {
      *reinterpret_cast<float4*>(o) = make_float4(v[0], v[1], v[2], v[3]);
    } else {
      for (int i = 0; i < 4 && x + i < w; ++i) o[i] = v[i];
    }
  };
  if (!box3) {
#pragma unroll
    for (int i = 0; i < kRgbRows; ++i) {
      if (y0 + i >= h) return;
      float g[6];
      gray6(y0 + i, g);
      put(y0 + i, {g[1], g[2], g[3], g[4]});
    }
    return;
  }
  // the prefilter leaves the frame's one-pixel border as it is
  float a[4], b[4], c[4], gb[4], gc[4];  // horizontal sums of rows y - 1, y, y + 1; gray of rows y, y + 1
  auto row = [&](int y, float (&hs)[4], float (&gr)[4]) {
    float g[6];
    gray6(min(max(y, 0), h - 1), g);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      hs[i] = box_h(g[i], g[i + 1], g[i + 2]);
      gr[i] = g[i + 1];
    }
  };
  row(y0 - 1, a, gb);
  row(y0, b, gb);
#pragma unroll
  for (int i = 0; i < kRgbRows; ++i) {
    const int y = y0 + i;
    if (y >= h) return;
    row(y + 1, c, gc);
    float v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const bool in = x + k > 0 && x + k < w - 1 && y > 0 && y < h - 1;
      v[k] = in ? box_v(a[k], b[k], c[k]) : gb[k];
    }
    put(y, v);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      a[k] = b[k];
      b[k] = c[k];
      gb[k] = gc[k];
    }
  }
}

}  // namespace

int l012_deep_floats() { return l012::kDeepFloats; }

int stage_tile(bool u8, int nl, int kt, bool lead) {
  if (u8 && nl == 2) return l012::kT2;
  if (lead && nl == 2) return lead::kT2;
  return (kt & 31) == 16 ? 16 : 8;
}

int lead_deep_max_width() { return lead::kDeepFloats / 8; }

namespace {

using TmapEncode = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// cuTensorMapEncodeTiled through the runtime's driver entry point, looked up once per process (the
// initialisation of a function-local static is thread-safe); null when unavailable.
TmapEncode tmap_encoder() {
  static const TmapEncode encode = []() -> TmapEncode {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      return reinterpret_cast<TmapEncode>(fn);
    return nullptr;
  }();
  return encode;
}

}  // namespace

bool encode_plane_tmap_f32(CUtensorMap* map, const float* base, int w, int h, int pitch_floats, int box_w, int box_h) {
  const TmapEncode encode = tmap_encoder();
  if (!encode || !map || !base || w <= 0 || h <= 0 || box_w <= 0 || box_h <= 0 || box_w > 256 || box_h > 256)
    return false;
  const int64_t pitch_bytes = (int64_t)pitch_floats * 4;
  if (((uintptr_t)base % 16) != 0 || (pitch_bytes % 16) != 0 || ((int64_t)box_w * 4) % 16 != 0) return false;
  const cuuint64_t dims[2] = {(cuuint64_t)w, (cuuint64_t)h};
  const cuuint64_t strides[1] = {(cuuint64_t)pitch_bytes};
  const cuuint32_t box[2] = {(cuuint32_t)box_w, (cuuint32_t)box_h};
  const cuuint32_t estr[2] = {1, 1};
  return encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(base), dims, strides, box, estr,
                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

bool encode_lead_tmap(StageJob& job) {
  // frames smaller than the box use plain copies
  job.use_tma = job.src_w >= lead::kW && job.src_h >= lead::kH && job.src_pitch_bytes % 16 == 0 &&
                encode_plane_tmap_f32(&job.tmap, static_cast<const float*>(job.src), job.src_w, job.src_h,
                                      (int)(job.src_pitch_bytes / 4), lead::kW, lead::kH);
  return job.use_tma != 0;
}

bool encode_frame_tmap(StageJob& job) {
  const TmapEncode encode = tmap_encoder();
  job.use_tma = 0;
  if (!encode) return false;
  // TMA needs a 16-byte aligned base and pitch; frames smaller than the box use plain loads
  if (((uintptr_t)job.src % 16) != 0 || (job.src_pitch_bytes % 16) != 0) return false;
  if (job.src_w < l012::kS0W || job.src_h < l012::kS0H) return false;
  const cuuint64_t dims[2] = {(cuuint64_t)job.src_w, (cuuint64_t)job.src_h};
  const cuuint64_t strides[1] = {(cuuint64_t)job.src_pitch_bytes};
  const cuuint32_t box[2] = {(cuuint32_t)l012::kS0W, (cuuint32_t)l012::kS0H};
  const cuuint32_t estr[2] = {1, 1};
  if (encode(&job.tmap, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(job.src), dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return false;
  job.use_tma = 1;
  return true;
}

namespace {
template <typename Batch>
cudaError_t set_l012_attrs() {
  cudaError_t e;
  const auto attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
  if ((e = cudaFuncSetAttribute(l012::pyramid_l012_kernel<2, Batch>, attr, l012::kSmemBox)) != cudaSuccess) return e;
  if ((e = cudaFuncSetAttribute(l012::pyramid_l012_kernel<3, Batch>, attr, l012::kSmemBox)) != cudaSuccess) return e;
  if ((e = cudaFuncSetAttribute(lead::pyramid_lead_kernel<Batch>, attr, lead::kSmem)) != cudaSuccess) return e;
  return cudaFuncSetAttribute(lead::pyramid_deep_kernel<Batch>, attr, lead::kDeepFloats * 4);
}

StageOne one_job(const StageBatch& b) {
  StageOne o;
  o.njobs = b.njobs;
  o.wait_limit = b.wait_limit;
  o.status = b.status;
  o.queue = b.queue;
  o.job[0] = b.job[0];
  return o;
}

template <typename Batch>
cudaError_t launch_l012(const Batch& b, int tiles, int kt, int smem, cudaStream_t s) {
  if (kt & kL012Three)
    l012::pyramid_l012_kernel<3, Batch><<<tiles, l012::kThreads, smem, s>>>(b);
  else
    l012::pyramid_l012_kernel<2, Batch><<<tiles, l012::kThreads, smem, s>>>(b);
  return cudaGetLastError();
}

template <typename Batch>
cudaError_t launch_lead(const Batch& b, int tiles, bool tail, cudaStream_t s) {
  lead::pyramid_lead_kernel<Batch><<<tiles, lead::kThreads, lead::kSmem, s>>>(b);
  if (tail)
    lead::pyramid_deep_kernel<Batch><<<b.njobs * lead::kDeepCtas, lead::kDeepThreads, lead::kDeepFloats * 4, s>>>(b);
  return cudaGetLastError();
}
}  // namespace

cudaError_t pyramid_init() {
  cudaError_t e;
  if ((e = set_l012_attrs<StageBatch>()) != cudaSuccess) return e;
  if ((e = set_l012_attrs<StageOne>()) != cudaSuccess) return e;
  if ((e = set_stage_attrs<8>()) != cudaSuccess) return e;
  return set_stage_attrs<16>();
}

cudaError_t launch_input_stage(const uint8_t* src, int64_t src_pitch, int channels, int box3, int w, int h,
                               float* dst, int64_t dst_pitch_floats, cudaStream_t s) {
  if (channels == 3) {
    const dim3 grid((w + 127) / 128, (h + 8 * kRgbRows - 1) / (8 * kRgbRows));
    input_rgb_kernel<<<grid, 256, 0, s>>>(src, src_pitch, box3, w, h, dst, dst_pitch_floats);
  } else {
    const dim3 block(32, 8), grid((w + 31) / 32, (h + 7) / 8);
    input_mono_kernel<<<grid, block, 0, s>>>(src, src_pitch, box3, w, h, dst, dst_pitch_floats);
  }
  return cudaGetLastError();
}

cudaError_t launch_pyramid_lead(const StageBatch& b, int tiles, bool tail, cudaStream_t s) {
  if (tiles <= 0) return cudaSuccess;
  return b.njobs == 1 ? launch_lead(one_job(b), tiles, tail, s) : launch_lead(b, tiles, tail, s);
}

cudaError_t launch_pyramid_stage(const StageBatch& b, int tiles, bool u8, int nl, int kt, bool tail, cudaStream_t s) {
  if (tiles <= 0) return cudaSuccess;
  if (u8) {
    switch (nl) {
      case 0: return launch_stage<uint8_t, 0>(b, tiles, kt, tail, s);
      case 1: return launch_stage<uint8_t, 1>(b, tiles, kt, tail, s);
      default:
        bool box = false;
        for (int j = 0; j < b.njobs; ++j) box = box || b.job[j].box3;
        const int smem = box ? l012::kSmemBox : l012::kSmem;
        return b.njobs == 1 ? launch_l012(one_job(b), tiles, kt, smem, s) : launch_l012(b, tiles, kt, smem, s);
    }
  }
  switch (nl) {
    case 0: return launch_stage<float, 0>(b, tiles, kt, tail, s);
    case 1: return launch_stage<float, 1>(b, tiles, kt, tail, s);
    default: return launch_stage<float, 2>(b, tiles, kt, tail, s);
  }
}

}  // namespace fe
