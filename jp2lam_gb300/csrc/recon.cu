// Decoder-side reconstruction of an encoded page on the device, for the
// quality metrics of jp2g_encode_with_psnr.
//
// Follows compute_quality_metrics (src/encode/backend/native/backend.rs:
// 305-433): each code-block's quantised coefficients are truncated to the
// last bit-plane its retained passes reach and dequantised at the midpoint
// (dequantize_truncated_coeff, backend.rs:628-639), the inverse 9/7 runs
// level by level, rows then columns (src/dwt/irrev97.rs:639-796), the
// inverse ICT and level shift give 8-bit samples (clamped), and the page's
// PSNR and mean 8x8 luma SSIM (mssim_8x8, backend.rs:911-959) come from
// them. Every f32 step is the reference's operation in its order without
// contraction (built with --fmad=false), so the reconstructed samples equal
// the oracle's; only the f64 sums run in a different order.
#include <cuda_runtime.h>

#include <type_traits>
#include <vector>

#include "jp2g_internal.h"
#include "kernels.h"

namespace jp2g {

namespace {

__constant__ float kRAlpha = -1.586134342059924f;
__constant__ float kRBeta = -0.052980118572961f;
__constant__ float kRGamma = 0.882911075530934f;
__constant__ float kRDelta = 0.443506852043971f;
__constant__ float kRK = 1.230174104914001f;
__constant__ float kRInvK = 1.0f / 1.230174104914001f;

// Whole-sample symmetric extension (src/dwt/irrev97.rs:523-536).
__device__ __forceinline__ int sym_at(int i, int n) {
  if (n <= 1) return 0;
  if (i >= 0 && i < n) return i;
  const int period = 2 * (n - 1);
  int k = i % period;
  if (k < 0) k += period;
  return k >= n ? period - k : k;
}

// Code-block samples -> midpoint dequantised f32 in the component's plane.
__global__ void recon_dequant_kernel(ReconArgs r) {
  const int lane = threadIdx.x & 31;
  const uint32_t b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (b >= r.nblocks) return;
  const BlockDesc d = r.blocks[b];
  const ReconBlock rb = r.rblocks[b];
  const uint32_t kept = r.keep[b].npasses;
  const int last_bp = kept ? r.passes[d.pass_off + kept - 1].bitplane : -1;
  const int32_t* q = r.coef + (size_t)d.coef_slot * r.cbw * r.cbh;
  float* out = r.plane + (size_t)rb.comp * r.width * r.height;
  for (int i = lane; i < d.w * d.h; i += 32) {
    const int y = i / d.w, x = i - y * d.w;
    const int32_t v = q[y * r.cbw + x];
    float o = 0.0f;
    if (last_bp >= 0) {
      const uint32_t a = v < 0 ? 0u - (uint32_t)v : (uint32_t)v;
      const uint32_t t = (a >> last_bp) << last_bp;
      if (t != 0) o = __fmul_rn(__fmul_rn(v >= 0 ? 1.0f : -1.0f, __fadd_rn((float)t, 0.5f)), rb.step);
    }
    out[(size_t)(rb.y0 + y) * r.width + rb.x0 + x] = o;
  }
}

__device__ __forceinline__ float lifted(float x, float c, float l, float rr) {
  return __fadd_rn(x, __fmul_rn(c, __fadd_rn(l, rr)));
}

// The job holding tile g of a level's launch.
__device__ __forceinline__ const IdwtJob& job_of(const IdwtJob* jobs, uint32_t njobs, uint32_t g) {
  uint32_t lo = 0, hi = njobs;
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (jobs[mid].tile_base <= g) lo = mid;
    else hi = mid;
  }
  return jobs[lo];
}

// One level of the inverse 2-D transform over 128x64 tiles, rows then
// columns:
//  9/7 (src/dwt/irrev97.rs:639-796): scale by K / 1/K, then four lifting
//    steps x[j] += c (x[j-1] + x[j+1]), each rounded as written;
//  5/3 (src/dwt/rev53.rs:96-129, 419-497): even samples
//    s[i] - ((d[i-1] + d[i] + 2) >> 2), then odd samples
//    d[i] + ((e[i] + e[i+1]) >> 1).
// A CTA loads a tile and 4 samples around it, interleaving the bands,
// positions beyond the region's ends from their mirror images: whole-sample
// symmetric extension commutes with each lifting step (a position and its
// mirror have the same parity and mirrored neighbours, and l + r = r + l
// exactly), so every output equals whole-row and whole-column lifting; the 5/3
// edge clamps are the same extension. A thread lifts 40 samples of a row, then
// of a column, in registers.
// A level is read once and written once (the samples beside a tile come from
// L2), into a buffer of its own, as neighbouring tiles still read the old
// bands. Bound by the latency of the loads at 4 CTAs per SM: 12 sRGB 2550x3300
// pages, all levels, 0.93 ms, the last one 0.66 (3.7 TB/s); a warp per row
// lifting in global memory, then column tiles, took 3.9, and loading sample by
// sample in place of pairs of columns 2.1.
constexpr int kTileW = kIdwtTileCols, kTileH = kIdwtTileRows, kHalo = 4;
constexpr int kSpanW = kTileW + 2 * kHalo, kSpanH = kTileH + 2 * kHalo, kPitch = kSpanW + 2;
constexpr int kJob = 40;  // samples of a register job: 32 outputs and a halo
constexpr int kIdwtThreads = 288, kWarps = kIdwtThreads / 32;
static_assert(kSpanH % kWarps == 0 && kSpanW / 2 > 64 && kSpanW / 2 <= 96, "rows and pairs of the load");
static_assert(kPitch % 4 == 2, "pairs are aligned and 32 rows' pairs lie in different banks");
static_assert(kIdwtThreads == kSpanH * (kTileW / 32) && kIdwtThreads >= kTileW * (kTileH / 32), "a job per thread");

template <class T>
struct alignas(8) Pair {
  T x, y;
};

// Outputs x[4..35] from x[1..39] (9/7) or x[3..37] (5/3), in place. single:
// the region is one sample long (only scaled).
__device__ __forceinline__ void unlift(float (&x)[kJob], bool single) {
  #pragma unroll
  for (int i = 1; i < kJob; ++i) x[i] = __fmul_rn(x[i], i & 1 ? kRInvK : kRK);
  if (single) return;
  #pragma unroll
  for (int i = 2; i <= 38; i += 2) x[i] = lifted(x[i], -kRDelta, x[i - 1], x[i + 1]);
  #pragma unroll
  for (int i = 3; i <= 37; i += 2) x[i] = lifted(x[i], -kRGamma, x[i - 1], x[i + 1]);
  #pragma unroll
  for (int i = 4; i <= 36; i += 2) x[i] = lifted(x[i], -kRBeta, x[i - 1], x[i + 1]);
  #pragma unroll
  for (int i = 5; i <= 35; i += 2) x[i] = lifted(x[i], -kRAlpha, x[i - 1], x[i + 1]);
}
__device__ __forceinline__ void unlift(int32_t (&x)[kJob], bool single) {
  if (single) return;
  #pragma unroll
  for (int i = 4; i <= 36; i += 2) x[i] -= (x[i - 1] + x[i + 1] + 2) >> 2;
  #pragma unroll
  for (int i = 5; i <= 35; i += 2) x[i] += (x[i - 1] + x[i + 1]) >> 1;
}

template <class T>
__device__ __forceinline__ void idwt_tile(const IdwtJob& jb, int x0, int y0, T* s) {
  const int tid = threadIdx.x, rw = (int)jb.rw, rh = (int)jb.rh;
  const int lw = (rw + 1) / 2, lh = (rh + 1) / 2;
  {
    // a warp per row: a lane's pairs of columns stay the same
    const T* ll = static_cast<const T*>(jb.ll);
    const T* detail = static_cast<const T*>(jb.detail);
    const int lane = tid & 31, warp = tid >> 5;
    int even[3], odd[3];  // where the pairs' samples lie in a row of bands
    bool mirrored[3];     // an odd position of a single column takes the even sample
    #pragma unroll
    for (int k = 0; k < 3; ++k) {
      const int j = x0 - kHalo + 2 * min(lane + 32 * k, kSpanW / 2 - 1);
      const int q = sym_at(j + 1, rw);
      even[k] = sym_at(j, rw) >> 1;
      odd[k] = (q & 1 ? lw : 0) + (q >> 1);
      mirrored[k] = !(q & 1);
    }
    #pragma unroll 4
    for (int i = 0; i < kSpanH / kWarps; ++i) {
      const int li = i * kWarps + warp, p = sym_at(y0 - kHalo + li, rh);
      const T* high = detail + (size_t)((p & 1 ? lh : 0) + (p >> 1)) * jb.detail_pitch;
      const T* low = p & 1 ? high : ll + (size_t)(p >> 1) * jb.ll_pitch;
      #pragma unroll
      for (int k = 0; k < 3; ++k)
        if (k < 2 || lane < kSpanW / 2 - 64) {
          Pair<T> v;
          v.x = low[even[k]];
          v.y = (mirrored[k] ? low : high)[odd[k]];
          *reinterpret_cast<Pair<T>*>(s + li * kPitch + 2 * (lane + 32 * k)) = v;
        }
    }
  }
  __syncthreads();
  T x[kJob];
  {
    const int row = tid % kSpanH, first = 32 * (tid / kSpanH);
    T* at = s + row * kPitch + first;
    #pragma unroll
    for (int i = 0; i < kJob; i += 2) {
      const Pair<T> v = *reinterpret_cast<const Pair<T>*>(at + i);
      x[i] = v.x;
      x[i + 1] = v.y;
    }
    __syncthreads();
    unlift(x, rw == 1);
    #pragma unroll
    for (int i = kHalo; i < kHalo + 32; i += 2) *reinterpret_cast<Pair<T>*>(at + i) = Pair<T>{x[i], x[i + 1]};
    const int end = rw - 1 - (x0 - kHalo + first);
    if (std::is_same<T, int32_t>::value && rw > 1 && !(rw & 1) && end >= kHalo && end < kHalo + 32) {
      // a row's last sample adds its even neighbour itself: half of its double
      // differs where a sample is too large to be doubled
      const int32_t e = at[end - 1];
      at[end] += e - ((int32_t)(2u * (uint32_t)e) >> 1);
    }
  }
  __syncthreads();
  if (tid >= kTileW * (kTileH / 32)) return;
  const int cx = x0 + tid % kTileW, first = 32 * (tid / kTileW);
  const T* at = s + first * kPitch + kHalo + tid % kTileW;
  #pragma unroll
  for (int i = 1; i < kJob; ++i) x[i] = at[i * kPitch];
  unlift(x, rh == 1);
  if (cx >= rw) return;
  T* out = static_cast<T*>(jb.out) + (size_t)(y0 + first) * jb.out_pitch + cx;
  #pragma unroll
  for (int i = 0; i < 32; ++i)
    if (y0 + first + i < rh) out[(size_t)i * jb.out_pitch] = x[kHalo + i];
}

__global__ void __launch_bounds__(kIdwtThreads) idwt_kernel(const IdwtJob* jobs, uint32_t njobs) {
  __shared__ alignas(16) float s[kSpanH * kPitch];
  const IdwtJob& jb = job_of(jobs, njobs, blockIdx.x);
  const uint32_t tiles_x = (jb.rw + kTileW - 1) / kTileW, t = blockIdx.x - jb.tile_base;
  const int x0 = (int)(t % tiles_x) * kTileW, y0 = (int)(t / tiles_x) * kTileH;
  if (jb.reversible) idwt_tile(jb, x0, y0, reinterpret_cast<int32_t*>(s));
  else idwt_tile(jb, x0, y0, s);
}

__device__ __forceinline__ float clamp255(float v) { return fminf(fmaxf(v, 0.0f), 255.0f); }

__device__ __forceinline__ double block_sum(double v, double* sh) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(~0u, v, o);
  const int w = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) sh[w] = v;
  __syncthreads();
  double s = 0;
  if (threadIdx.x == 0)
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) s += sh[i];
  return s;
}

// Decoded samples: squared error against the original pixels, and the
// original and decoded luma (BT.601 for sRGB) for SSIM.
__global__ void recon_pixels_kernel(ReconArgs r) {
  __shared__ double sh[8];
  const size_t n = (size_t)r.width * r.height;
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  double e = 0.0;
  if (i < n) {
    if (r.ncomp == 1) {
      const float dec = clamp255(__fadd_rn(r.samples[i], 128.0f));
      const float orig = (float)r.px[i];
      const float diff = __fadd_rn(dec, -orig);
      e = (double)__fmul_rn(diff, diff);
      r.luma_dec[i] = dec;
      r.luma_orig[i] = orig;
    } else {
      const float yc = r.samples[i], cb = r.samples[n + i], cr = r.samples[2 * n + i];
      // inverse ICT (ISO/IEC 15444-1 G.2) and level shift, backend.rs:392-400
      const float R = clamp255(__fadd_rn(__fadd_rn(yc, __fmul_rn(1.402f, cr)), 128.0f));
      const float G = clamp255(
          __fadd_rn(__fadd_rn(__fadd_rn(yc, -__fmul_rn(0.34413f, cb)), -__fmul_rn(0.71414f, cr)), 128.0f));
      const float B = clamp255(__fadd_rn(__fadd_rn(yc, __fmul_rn(1.772f, cb)), 128.0f));
      const float o0 = (float)r.px[3 * i], o1 = (float)r.px[3 * i + 1], o2 = (float)r.px[3 * i + 2];
      const float dr = __fadd_rn(R, -o0), dg = __fadd_rn(G, -o1), db = __fadd_rn(B, -o2);
      e = (double)__fadd_rn(__fadd_rn(__fmul_rn(dr, dr), __fmul_rn(dg, dg)), __fmul_rn(db, db));
      r.luma_dec[i] = __fadd_rn(__fadd_rn(__fmul_rn(0.299f, R), __fmul_rn(0.587f, G)), __fmul_rn(0.114f, B));
      r.luma_orig[i] = __fadd_rn(__fadd_rn(__fmul_rn(0.299f, o0), __fmul_rn(0.587f, o1)), __fmul_rn(0.114f, o2));
    }
  }
  const double s = block_sum(e, sh);
  if (threadIdx.x == 0) atomicAdd(&r.stats[0], s);
}

// SSIM of one 8x8 luma block per thread (sums in the reference's order).
__global__ void recon_ssim_kernel(ReconArgs r) {
  __shared__ double sh[8];
  const int bc = r.width / 8, br = r.height / 8;
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  double v = 0.0;
  if (k < bc * br) {
    const int by = k / bc, bx = k - by * bc;
    double sx = 0, sy = 0, sxx = 0, syy = 0, sxy = 0;
    for (int dy = 0; dy < 8; ++dy)
      for (int dx = 0; dx < 8; ++dx) {
        const size_t i = (size_t)(by * 8 + dy) * r.width + bx * 8 + dx;
        const double x = r.luma_orig[i], y = r.luma_dec[i];
        sx = __dadd_rn(sx, x);
        sy = __dadd_rn(sy, y);
        sxx = __dadd_rn(sxx, __dmul_rn(x, x));
        syy = __dadd_rn(syy, __dmul_rn(y, y));
        sxy = __dadd_rn(sxy, __dmul_rn(x, y));
      }
    const double n = 64.0, C1 = 6.5025, C2 = 58.5225;
    const double ux = __ddiv_rn(sx, n), uy = __ddiv_rn(sy, n);
    const double vx = fmax(__dadd_rn(__ddiv_rn(sxx, n), -__dmul_rn(ux, ux)), 0.0);
    const double vy = fmax(__dadd_rn(__ddiv_rn(syy, n), -__dmul_rn(uy, uy)), 0.0);
    const double cxy = __dadd_rn(__ddiv_rn(sxy, n), -__dmul_rn(ux, uy));
    const double num = __dmul_rn(__dadd_rn(__dmul_rn(__dmul_rn(2.0, ux), uy), C1), __dadd_rn(__dmul_rn(2.0, cxy), C2));
    const double den = __dmul_rn(__dadd_rn(__dadd_rn(__dmul_rn(ux, ux), __dmul_rn(uy, uy)), C1),
                                 __dadd_rn(__dadd_rn(vx, vy), C2));
    v = __ddiv_rn(num, den);
  }
  const double s = block_sum(v, sh);
  if (threadIdx.x == 0) atomicAdd(&r.stats[1], s);
}

// ------------------------------------------------------------- decoding --
__device__ __forceinline__ uint32_t clamp_int(int32_t v) { return (uint32_t)min(max(v + 128, 0), 255); }
__device__ __forceinline__ uint32_t clamp_round(float v) {
  return (uint32_t)(int)fminf(fmaxf(roundf(__fadd_rn(v, 128.0f)), 0.0f), 255.0f);
}

// Inverse RCT (src/simd/scalar.rs:216-228) or ICT (scalar.rs:201-214), the
// level shift and clamp (finalize, scalar.rs:230-242) of sample i of a page of n,
// as bytes from bit 0 on.
__device__ __forceinline__ uint32_t pixel_of(const PixJob& jb, int32_t s0, int32_t s1, int32_t s2) {
  if (jb.reversible) {
    if (jb.mct) {
      const int32_t gg = s0 - ((s1 + s2) >> 2);
      return clamp_int(s2 + gg) | clamp_int(gg) << 8 | clamp_int(s1 + gg) << 16;
    }
    return clamp_int(s0) | clamp_int(s1) << 8 | clamp_int(s2) << 16;
  }
  const float yy = __int_as_float(s0), cb = __int_as_float(s1), cr = __int_as_float(s2);
  if (jb.mct)
    return clamp_round(__fadd_rn(yy, __fmul_rn(1.402f, cr))) |
           clamp_round(__fadd_rn(__fadd_rn(yy, -__fmul_rn(0.34413f, cb)), -__fmul_rn(0.71414f, cr))) << 8 |
           clamp_round(__fadd_rn(yy, __fmul_rn(1.772f, cb))) << 16;
  return clamp_round(yy) | clamp_round(cb) << 8 | clamp_round(cr) << 16;
}

// A page's samples, written interleaved: a CTA takes kPixBlock of them, a
// thread four in a row by 16-byte loads and 4-byte stores where the planes and
// the output are aligned for them, else every 256th. Bound by memory: 12 sRGB
// 2550x3300 pages 0.22 ms; a thread per sample, by byte stores, took 0.49.
__global__ void __launch_bounds__(256) dec_pixels_kernel(const PixJob* jobs, uint32_t njobs) {
  uint32_t lo = 0, hi = njobs;
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (jobs[mid].block_base <= blockIdx.x) lo = mid;
    else hi = mid;
  }
  const PixJob jb = jobs[lo];
  const size_t n = jb.npx, first = (size_t)(blockIdx.x - jb.block_base) * kPixBlock;
  const int32_t* q = jb.planes;
  const bool aligned = n % 4 == 0 && reinterpret_cast<size_t>(q) % 16 == 0 && reinterpret_cast<size_t>(jb.px) % 4 == 0;
  if (aligned) {
    const size_t i = first + 4 * threadIdx.x;
    if (i >= n) return;
    const int4 z = make_int4(0, 0, 0, 0);
    const int4 s0 = *reinterpret_cast<const int4*>(q + i);
    const int4 s1 = jb.ncomp == 3 ? *reinterpret_cast<const int4*>(q + n + i) : z;
    const int4 s2 = jb.ncomp == 3 ? *reinterpret_cast<const int4*>(q + 2 * n + i) : z;
    const uint32_t p0 = pixel_of(jb, s0.x, s1.x, s2.x), p1 = pixel_of(jb, s0.y, s1.y, s2.y);
    const uint32_t p2 = pixel_of(jb, s0.z, s1.z, s2.z), p3 = pixel_of(jb, s0.w, s1.w, s2.w);
    uint32_t* out = reinterpret_cast<uint32_t*>(jb.px + jb.ncomp * i);
    if (jb.ncomp == 3) {
      out[0] = p0 | p1 << 24;
      out[1] = p1 >> 8 | p2 << 16;
      out[2] = p2 >> 16 | p3 << 8;
    } else {
      out[0] = (p0 & 0xffu) | (p1 & 0xffu) << 8 | (p2 & 0xffu) << 16 | p3 << 24;
    }
    return;
  }
  #pragma unroll
  for (uint32_t k = 0; k < kPixBlock; k += 256) {
    const size_t i = first + k + threadIdx.x;
    if (i >= n) return;
    const bool three = jb.ncomp == 3;
    const uint32_t p = pixel_of(jb, q[i], three ? q[n + i] : 0, three ? q[2 * n + i] : 0);
    uint8_t* out = jb.px + jb.ncomp * i;
    out[0] = (uint8_t)p;
    if (three) {
      out[1] = (uint8_t)(p >> 8);
      out[2] = (uint8_t)(p >> 16);
    }
  }
}

}  // namespace

uint32_t idwt_tiles(uint32_t rw, uint32_t rh) {
  return ((rw + kIdwtTileCols - 1) / kIdwtTileCols) * ((rh + kIdwtTileRows - 1) / kIdwtTileRows);
}

// Jobs of one component, smallest level first. Level l reads its LL band
// from where level l - 1 left it (the plane's own corner at first) and its
// other bands from the plane, and writes whole samples to `out` or `other` in
// turn, so that the last level's come to `out`.
void idwt_jobs(void* plane, void* out, void* other, const std::pair<int, int>* ladder, int levels, bool reversible,
               std::vector<std::vector<IdwtJob>>* by_level) {
  const uint32_t width = (uint32_t)ladder[levels].first;
  const void* ll = plane;
  uint32_t ll_pitch = width;
  for (int l = 1; l <= levels; ++l) {
    const uint32_t rw = (uint32_t)ladder[l].first, rh = (uint32_t)ladder[l].second;
    if (rw == 0 || rh == 0) continue;
    IdwtJob j{};
    j.detail = plane;
    j.detail_pitch = width;
    j.ll = ll;
    j.ll_pitch = ll_pitch;
    j.out = (levels - l) % 2 == 0 ? out : other;
    j.out_pitch = rw;
    j.rw = rw;
    j.rh = rh;
    j.reversible = reversible ? 1u : 0u;
    ll = j.out;
    ll_pitch = rw;
    (*by_level)[l].push_back(j);
  }
}

void launch_idwt_level(const IdwtJob* jobs, uint32_t njobs, uint32_t total_tiles, cudaStream_t st) {
  if (njobs == 0 || total_tiles == 0) return;
  idwt_kernel<<<total_tiles, kIdwtThreads, 0, st>>>(jobs, njobs);
}

void launch_dec_pixels(const PixJob* jobs, uint32_t njobs, uint32_t nblocks, cudaStream_t st) {
  if (njobs == 0 || nblocks == 0) return;
  dec_pixels_kernel<<<nblocks, 256, 0, st>>>(jobs, njobs);
}

void launch_recon(ReconArgs r, const std::pair<int, int>* ladder, int levels, cudaStream_t st) {
  const size_t n = (size_t)r.width * r.height;
  cudaMemsetAsync(r.plane, 0, n * r.ncomp * sizeof(float), st);
  cudaMemsetAsync(r.stats, 0, 2 * sizeof(double), st);
  if (r.nblocks) recon_dequant_kernel<<<(unsigned)(((size_t)r.nblocks * 32 + 255) / 256), 256, 0, st>>>(r);
  // every component of a level in one launch; the levels alternate between
  // tmp and the luma planes, which are made only afterwards, and end in tmp
  std::vector<std::vector<IdwtJob>> by_level(levels + 1);
  const size_t half = (size_t)((r.width + 1) / 2) * ((r.height + 1) / 2);
  for (int c = 0; c < r.ncomp; ++c)
    idwt_jobs(r.plane + (size_t)c * n, r.tmp + (size_t)c * n, r.luma_orig + (size_t)c * half, ladder, levels, false,
              &by_level);
  std::vector<IdwtJob> jobs;
  std::vector<uint32_t> first(levels + 2, 0), tiles(levels + 1, 0);
  for (int l = 1; l <= levels; ++l) {
    first[l] = (uint32_t)jobs.size();
    for (IdwtJob j : by_level[l]) {
      j.tile_base = tiles[l];
      tiles[l] += idwt_tiles(j.rw, j.rh);
      jobs.push_back(j);
    }
  }
  first[levels + 1] = (uint32_t)jobs.size();
  if (!jobs.empty()) cudaMemcpyAsync(r.jobs, jobs.data(), jobs.size() * sizeof(IdwtJob), cudaMemcpyHostToDevice, st);
  for (int l = 1; l <= levels; ++l) launch_idwt_level(r.jobs + first[l], first[l + 1] - first[l], tiles[l], st);
  r.samples = levels > 0 ? r.tmp : r.plane;
  recon_pixels_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(r);
  const int nb8 = (int)(r.width / 8) * (int)(r.height / 8);
  if (nb8 > 0) recon_ssim_kernel<<<(unsigned)((nb8 + 255) / 256), 256, 0, st>>>(r);
}

}  // namespace jp2g
