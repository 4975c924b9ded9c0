// EBCOT Tier-1 encoder, single MQ termination per code-block, per-pass
// numbytes() snapshots for rate control.
//
// Replaces analyze_codeblock (src/encode/backend/native/t1.rs:215-258) and
// encode_codeblock_single_term (t1.rs:508-658) with its passes (SP
// t1.rs:805-905, MR t1.rs:914-965, cleanup t1.rs:977-1197) and the MQ coder
// (src/mq/mod.rs:163-432).
//
// The work is split where the dependencies allow:
//
// 1. t1_analyze_kernel (warp per block): max magnitude, non-zero count ->
//    magnitude bit-planes, zero bit-planes, block class.
//    t1_planes_kernel (warp per block): column masks per bit-plane, and from
//    their counts which bit-planes to model and how many symbols to expect;
//    t1_split_kernel: the blocks with the most, to be modelled and coded first.
// 2. t1_model_kernel (warp per (block, bit-plane)): the significance state
//    at the start of bit-plane p is known in closed form (|q| >> (p+1) != 0),
//    and so is the refinement history (|q| >> (p+2) != 0), so every
//    bit-plane's three passes are modelled independently. Within a
//    bit-plane, significance propagation is the least fixpoint of a
//    monotone system over 64-bit row masks in which each sample only looks
//    at samples earlier in the scan order (stripe by stripe); refinement and
//    cleanup are then data-parallel. The warp emits the (context, bit)
//    symbols of each stripe in exact scan order with a prefix sum over the
//    columns (one lane per column), into a per-bit-plane symbol slot.
// 3. t1_mq_kernel (lane per block): runs the MQ coder over a block's symbol
//    streams, top bit-plane first, recording numbytes() after every pass
//    and writing the byte stream to the block's payload slot, until rate
//    control can choose none of the passes to come (Stop).
#include <cuda_runtime.h>

#include <algorithm>

#include "jp2g_internal.h"
#include "kernels.h"
#include "t1_logic.h"

namespace jp2g {

namespace {

// Context numbers (src/mq/mod.rs:5-10).
constexpr int kCtxAGG = 17, kCtxUNI = 18;
constexpr uint32_t kCtxNone = 19;               // a context of Qe 0: coding its symbols changes nothing
constexpr uint32_t kPadSymbol = kCtxNone;  // pads symbol streams to whole chunks
// A symbol is a byte: context | decision << 7.
constexpr uint32_t kOne = 0x80u;
constexpr uint32_t kMqCtx = 20;
constexpr int kModelWarps = 4;  // 7 KB of shared memory each; registers allow 5 CTAs per SM
constexpr int kMqWarps = 4;

// The MQ states, qe | nmps << 16 | nlps << 24: built on the host from the
// standard's rules, copied in by upload_t1_tables. (The context rules are logic
// operations, t1_logic.h.)
constexpr uint32_t kStates = 94;
__constant__ uint32_t c_mq[kStates];

// ---------------------------------------------------------------- analyze --
// A warp per block, 16 bytes a lane, eight loads in flight. Bound by memory in
// large waves and by the loads' latency in small ones: a 256x256 page 8.9 us, 31
// with 4-byte loads, two at a time.
__global__ void __launch_bounds__(256) t1_analyze_kernel(T1Args a) {
  const int lane = threadIdx.x & 31;
  const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (warp >= a.nblocks) return;
  const BlockDesc d = a.blocks[warp];
  const int w = d.w, h = d.h;
  // lane l takes four columns of rows l / quads, + 32 / quads, ...
  const int quads = a.cbw / 4, x = 4 * (lane % quads), step = 32 / quads;
  const int4* src = reinterpret_cast<const int4*>(a.coef + (size_t)d.coef_slot * a.cbw * a.cbh) + lane;
  uint32_t mx = 0, nnz = 0;
  auto count = [&](int32_t v, bool in) {
    v = in ? v : 0;
    mx = max(mx, v < 0 ? 0u - (uint32_t)v : (uint32_t)v);
    nnz += v != 0;
  };
  for (int y = lane / quads; y - lane / quads < h; y += 8 * step, src += 8 * 32) {
    int4 v[8];  // (rows past the block's lie in its slot)
    #pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = src[k * 32];
    #pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int in = y + k * step < h ? w : 0;
      count(v[k].x, x < in);
      count(v[k].y, x + 1 < in);
      count(v[k].z, x + 2 < in);
      count(v[k].w, x + 3 < in);
    }
  }
  mx = __reduce_max_sync(0xffffffffu, mx);
  nnz = __reduce_add_sync(0xffffffffu, nnz);
  if (lane != 0) return;
  const int mbp = mx == 0 ? 0 : 32 - __clz(mx);
  // classify_from_nonzero_fraction (src/profile.rs:122-130), in f32.
  const float frac = __fdiv_rn((float)nnz, (float)(w * h));
  BlockOut o{};
  o.mbp = (uint8_t)mbp;
  o.zbp = (uint8_t)(d.mb > mbp ? d.mb - mbp : 0);
  o.cls = (uint8_t)(mbp == 0 ? 0 : (frac <= 0.05f ? 0 : (frac <= 0.30f ? 1 : 2)));
  uint32_t np = mbp == 0 ? 0u : 1u + 3u * (uint32_t)(mbp - 1);
  o.status = np > a.pass_cap ? 2 : 0;
  o.npasses = o.status ? 0 : (uint16_t)np;
  a.res[warp] = o;
  a.nplanes[warp] = o.status ? 0u : (uint32_t)mbp;
}

// Distortion of one significant sample of a block at bit-plane 0: the
// weights of pcrd_hull_kernel in f32.
__device__ __forceinline__ float block_unit(const T1Args& a, uint32_t b, const BlockDesc& d) {
  const BandParam& bp = a.bands[d.band_param];
  const uint32_t cls = a.res[b].cls;
  const float base = cls == 0 ? 2.5f : (cls == 1 ? 1.5f : 1.0f);
  return bp.unit * (bp.is_ll ? base * 1.1f : base) * a.comps[d.comp_key].weight;
}

constexpr uint32_t kHeavy = 0x80000000u;  // T1Args::weight

// 4^k: the energy of bit-plane k against bit-plane 0's (capped as in pcrd.cu).
__device__ __forceinline__ float plane_energy(int k) { return __uint_as_float((uint32_t)(127 + 2 * min(k, 30)) << 23); }

// One warp per code-block: lists the block's items and writes, for every
// bit-plane p it codes, the column masks the modelling kernel starts from:
// significant before the plane (|q| >> (p+1) != 0) and the magnitude bit p,
// plus the block's sign masks. A lane reads 32 rows of one column, and a
// transpose in registers turns 32 magnitudes into 32 bit-plane masks, so
// every coefficient is read once per block instead of once per plane.
// Layout: planes[((item * 2 + {0: S, 1: B}) * 2 + half) * 64 + column],
// signs[(block * 2 + half) * 64 + column], half 0 = rows 0-31.
// Bound by the latency of its loads and stores: with 64 registers four CTAs fit
// an SM in place of the two that 102 left
// (1.2 -> 0.77 ms for 24 sRGB 2550x3300 pages; three CTAs: 0.85).
__global__ void __launch_bounds__(256, 4) t1_planes_kernel(T1Args a) {
  const int lane = threadIdx.x & 31;
  const uint32_t b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (b >= a.nblocks) return;
  const uint32_t np = a.nplanes[b], base = a.plane_base[b];
  const BlockDesc d = a.blocks[b];
  const int w = d.w, h = d.h, mbp = (int)np;
  const int32_t* blk = a.coef + (size_t)d.coef_slot * a.cbw * a.cbh;
  uint32_t first[8] = {};  // per bit-plane, a byte: samples whose top bit it is
  #pragma unroll 1
  for (int col = 0; col < 2; ++col) {
    const int x = lane + 32 * col;
    #pragma unroll 1
    for (int half = 0; half < 2; ++half) {
      uint32_t t[32], sg = 0;
      #pragma unroll
      for (int i = 0; i < 32; ++i) {
        const int y = 32 * half + i;
        const int32_t q = y < h && x < w ? blk[y * a.cbw + x] : 0;
        t[i] = q < 0 ? 0u - (uint32_t)q : (uint32_t)q;
        sg |= q < 0 ? 1u << i : 0u;
      }
      a.signs[((size_t)b * 2 + half) * 64 + x] = sg;
      if (mbp == 0) continue;
      transpose32(t);
      uint32_t above = 0;  // rows with a bit above plane k
      #pragma unroll
      for (int k = 31; k >= 0; --k) {
        if (k < mbp) {
          const size_t item = base + (uint32_t)(mbp - 1 - k);
          a.planes[((item * 2 + 0) * 2 + half) * 64 + x] = above;
          a.planes[((item * 2 + 1) * 2 + half) * 64 + x] = t[k];
        }
        first[k >> 2] += (uint32_t)__popc(t[k] & ~above) << (8 * (k & 3));  // at most 4 x 32
        above |= t[k];
      }
    }
  }
  if (mbp == 0) {
    if (lane == 0 && a.weight) a.weight[b] = 0;
    return;
  }
  // ItemRec::remain, by the distortion model of rate control (pcrd.cu), with
  // every newly significant sample taken as coded in significance propagation
  // (weight 1, cleanup has 0.85). Lane k holds bit-plane k.
  uint32_t newly = 0;
  #pragma unroll
  for (int k = 0; k < 32; ++k) {
    const uint32_t n = __reduce_add_sync(0xffffffffu, (first[k >> 2] >> (8 * (k & 3))) & 0xffu);
    if (lane == k) newly = n;
  }
  uint32_t sig = newly;  // samples significant at bit-plane k or above
  #pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t v = __shfl_down_sync(0xffffffffu, sig, o);
    if (lane + o < 32) sig += v;
  }
  const float gain = ((float)newly + 0.25f * (float)(sig - newly)) * plane_energy(lane);
  float below = lane < mbp ? gain : 0.0f;  // planes 0..k
  #pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const float v = __shfl_up_sync(0xffffffffu, below, o);
    if (lane >= o) below += v;
  }
  below = __shfl_up_sync(0xffffffffu, below, 1);  // planes 0..k-1
  const float unit = block_unit(a, b, d);
  if (lane < mbp)
    a.item_rec[base + (uint32_t)(mbp - 1 - lane)].remain = lane == 0 ? 0.0f : below * unit * 1.00001f;
  // The bit-planes to model: to the one after which coding is likely to stop
  // (see Stop), and one more. Bytes are estimated from the counts: a sample
  // that may become significant costs the entropy of doing so, less a share
  // for its context, and a sign; one already significant nearly a bit.
  // On a 2550x3300 page 2 blocks of 2,107 need more than that.
  uint32_t count = (uint32_t)mbp;
  const CompParam& cp = a.comps[d.comp_key];
  if (a.foresee && !cp.lossless) {
    const float before = (float)(sig - newly), open = (float)(w * h) - before, n = (float)newly;
    const float p = open > 0.0f ? n / open : 0.0f;
    const float entropy = p > 0.0f && p < 1.0f ? -(p * __log2f(p) + (1.0f - p) * __log2f(1.0f - p)) : 0.0f;
    float bytes = lane < mbp ? (0.7f * open * entropy + n + 0.9f * before) * 0.125f : 0.0f;
    float removed = lane < mbp ? gain * unit : 0.0f;
    #pragma unroll
    for (int o = 1; o < 32; o <<= 1) {  // planes k and above
      const float vb = __shfl_down_sync(0xffffffffu, bytes, o), vr = __shfl_down_sync(0xffffffffu, removed, o);
      if (lane + o < 32) {
        bytes += vb;
        removed += vr;
      }
    }
    const float value = removed - cp.lambda * (bytes + 2.0f);
    float best = lane < mbp ? fmaxf(value, 0.0f) : 0.0f;
    #pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float v = __shfl_down_sync(0xffffffffu, best, o);
      if (lane + o < 32) best = fmaxf(best, v);
    }
    const float rest = lane == 0 ? 0.0f : below * unit;
    const uint32_t stops = __ballot_sync(0xffffffffu, lane < mbp && value + rest < best);
    if (stops) count = min(count, (uint32_t)(mbp - (31 - __clz((int)stops))) + 1u);
  }
  if (lane == 0) a.nplanes[b] = count;
  if (a.weight) {
    // symbols: a refinement or a sign each, and a zero coding of every sample
    // near a significant one, of a quarter of the others
    const uint32_t open = (uint32_t)(w * h) - (sig - newly), near = min(open, 6u * sig);
    const bool coded = lane < mbp && lane >= mbp - (int)count;
    const uint32_t n = __reduce_add_sync(0xffffffffu, coded ? sig + near + (open - near) / 4u : 0u);
    if (lane == 0) {
      a.weight[b] = n | (a.bands[d.band_param].is_ll ? kHeavy : 0u);
      if (n > *const_cast<volatile uint32_t*>(a.counts + kCountWeight)) atomicMax(a.counts + kCountWeight, n);
    }
    return;
  }
  uint32_t at = 0;
  if (lane == 0) at = atomicAdd(a.counts + kCountItems, count);
  at = __shfl_sync(0xffffffffu, at, 0);
  for (uint32_t j = lane; j < count; j += 32) a.items[at + j] = b << 6 | j;
}

// The part of a block in a split wave: 0 from a share of the largest expected
// symbol count on (and LL bands: few, and the ones whose slopes settle their
// components' lambda), 1 below.
__device__ __forceinline__ int part_of(const T1Args& a, uint32_t b) {
  const uint32_t v = a.weight[b];
  return v >= kHeavy || 12u * v >= a.share * a.counts[kCountWeight] ? 0 : 1;
}

// A thread per block: counts the parts' blocks and lists their items.
__global__ void __launch_bounds__(256) t1_split_kernel(T1Args a) {
  const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31;
  const int part = b < a.nblocks ? part_of(a, b) : -1;
  const uint32_t n = part >= 0 ? a.nplanes[b] : 0u;
  uint32_t at = 0;
  #pragma unroll
  for (int p = 0; p < kT1Parts; ++p) {
    const uint32_t blocks = __ballot_sync(0xffffffffu, part == p);
    if (blocks == 0) continue;
    uint32_t sum = part == p ? n : 0u;
    #pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(0xffffffffu, sum, o);
      if (lane >= o) sum += v;
    }
    uint32_t first = 0;
    if (lane == 31) {
      first = atomicAdd(a.counts + kCountItems + p, sum);
      atomicAdd(a.counts + kCountBlocks + p, (uint32_t)__popc(blocks));
    }
    first = __shfl_sync(0xffffffffu, first, 31);
    if (part == p) at = p * a.nitems + first + sum - n;
  }
  for (uint32_t j = 0; j < n; ++j) a.items[at + j] = b << 6 | j;
}

// Modelling works on the code-block in column layout: lane L owns columns
// L ("A") and L + 32 ("B"), and every per-sample state of a column is a
// 64-bit mask with bit y = row y. Vertical neighbours are then shifts of the
// lane's own masks, horizontal ones a shuffle from the adjacent lane, and one
// logic operation handles 64 samples.
constexpr uint64_t kRow0 = 0x1111111111111111ull;  // first row of each stripe
constexpr uint64_t kRow3 = 0x8888888888888888ull;  // last row of each stripe

__device__ __forceinline__ uint64_t shfl64(uint64_t v, int src) {
  const uint32_t lo = __shfl_sync(~0u, (uint32_t)v, src);
  const uint32_t hi = __shfl_sync(~0u, (uint32_t)(v >> 32), src);
  return (uint64_t)hi << 32 | lo;
}

// The masks of the columns west and east of this lane's columns A and B.
struct Side {
  uint64_t wa, ea, wb, eb;
};
__device__ __forceinline__ Side sides(uint64_t a, uint64_t b, int lane) {
  const int up = (lane + 31) & 31, dn = (lane + 1) & 31;
  Side r;
  r.wa = shfl64(a, up);                   // column L - 1 (none for lane 0)
  r.wb = shfl64(lane == 31 ? a : b, up);  // column L + 31 (lane 0: column 31)
  r.ea = shfl64(lane == 0 ? b : a, dn);   // column L + 1 (lane 31: column 32)
  r.eb = shfl64(b, dn);                   // column L + 33 (none for lane 31)
  if (lane == 0) r.wa = 0;
  if (lane == 31) r.eb = 0;
  return r;
}

// Neighbourhood of every sample of a column at the moment it is coded in a
// pass: samples coded earlier in the pass (the column to the west, the row
// above in the same column, and the row above the stripe) in their state
// after it (f), the others in their state before it (p); the row below the
// stripe is taken before the pass. fc/pc: this column; fw/pw: the column to
// the west; fe/pe: to the east.
struct Hood {
  uint64_t nw, n, ne, w, e, sw, s, se;
};
__device__ __forceinline__ Hood hood(uint64_t fc, uint64_t pc, uint64_t fw, uint64_t pw, uint64_t fe, uint64_t pe) {
  Hood h;
  h.n = fc << 1;
  h.s = pc >> 1;
  h.w = fw;
  h.e = pe;
  h.nw = fw << 1;
  h.ne = ((pe << 1) & ~kRow0) | ((fe << 1) & kRow0);
  h.sw = ((fw >> 1) & ~kRow3) | ((pw >> 1) & kRow3);
  h.se = pe >> 1;
  return h;
}

__device__ __forceinline__ uint64_t pick(uint64_t m, uint64_t a, uint64_t b) { return (a & m) | (b & ~m); }

// Symbol planes of one column: which pass codes each sample, its primary
// symbol (context << 1 | magnitude bit) and its sign symbol, as bit-planes.
enum Plane {
  kPlV = 0,   // coded in significance propagation
  kPlS,       // coded in magnitude refinement (significant before the plane)
  kPlC,       // coded in cleanup
  kPlB,       // magnitude bit of the plane
  kPlClean,   // bit 4s: the column's part of stripe s is a cleanup run
  kPlP0,      // primary context, bits 0..4
  kPlP1,
  kPlP2,
  kPlP3,
  kPlP4,
  kPlM0,      // sign context - 8, bits 0..2
  kPlM1,
  kPlM2,
  kPlX,       // sign ^ sign prediction
  kNumPlanes
};

// Shared memory of one warp: the planes of its 64 columns, split in the
// 32-bit halves of rows 0-31 and 32-63 (bank-conflict-free per half).
struct ModelSmem {
  uint32_t pl[kNumPlanes][2][64];
};

// Nibble (4 rows of stripe s) of a half-plane, s counted within the half.
__device__ __forceinline__ uint32_t nib(uint32_t v, int s) { return (v >> (4 * s)) & 0xfu; }
// The 4 bits of a nibble spread to bit 0 of each byte.
__device__ __forceinline__ uint32_t spread4(uint32_t n) { return (n * 0x00204081u) & 0x01010101u; }

// Symbols of one column of one stripe: the column's counts per pass.
__device__ __forceinline__ uint32_t column_counts(uint32_t v, uint32_t sm, uint32_t c, uint32_t b, uint32_t cl) {
  const uint32_t sp = __popc(v) + __popc(v & b), mr = __popc(sm);
  uint32_t cln;
  if (cl) {
    if (b == 0) {
      cln = 1;
    } else {
      const uint32_t after = 0xfu & ~((2u << (__ffs(b) - 1)) - 1u);
      cln = 4 + __popc(after) + __popc(after & b);
    }
  } else {
    cln = __popc(c) + __popc(c & b);
  }
  return sp | (mr << 11) | (cln << 21);
}

// Exclusive prefix of v over the warp's lanes; *total = the warp's sum.
__device__ __forceinline__ uint32_t warp_offset(uint32_t v, int lane, uint32_t* total) {
  uint32_t x = v;
  #pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += t;
  }
  *total = __shfl_sync(0xffffffffu, x, 31);
  return x - v;
}

// A pass's symbols fill whole 16-byte chunks of its item's slot.
__device__ __forceinline__ uint32_t pad16(uint32_t n) { return (n + 15u) & ~15u; }

// Writes the symbols of one column of one stripe into the three streams.
__device__ __forceinline__ void emit_column(uint32_t v, uint32_t sm, uint32_t c, uint32_t b, uint32_t cl,
                                            uint32_t prim, uint32_t sgn, uint8_t*& osp, uint8_t*& omr,
                                            uint8_t*& ocl) {
  int first = 0;  // rows consumed by a cleanup run
  if (cl) {
    if (b == 0) {
      *ocl++ = (uint8_t)kCtxAGG;
      first = 4;
    } else {
      const int rl = __ffs(b) - 1;
      ocl[0] = (uint8_t)(kCtxAGG | kOne);
      ocl[1] = (uint8_t)(kCtxUNI | ((uint32_t)rl >> 1) << 7);
      ocl[2] = (uint8_t)(kCtxUNI | ((uint32_t)rl & 1u) << 7);
      ocl[3] = (uint8_t)(sgn >> (8 * rl));  // sign of the run's first significant sample
      ocl += 4;
      first = rl + 1;
    }
  }
  // every row in the same predicated code: the lanes of a warp code
  // samples of different passes at the same row
  #pragma unroll
  for (int r = 0; r < 4; ++r) {
    const uint32_t bit = (b >> r) & 1u;
    const bool im = (sm >> r) & 1u;
    const bool iv = (v >> r) & 1u;
    const bool ic = r >= first && ((c >> r) & 1u);
    uint8_t* o = im ? omr : (iv ? osp : ocl);
    if (im | iv | ic) o[0] = (uint8_t)(prim >> (8 * r));
    if ((iv | ic) && bit) o[1] = (uint8_t)(sgn >> (8 * r));
    omr += im ? 1 : 0;
    osp += iv ? 1 + bit : 0;
    ocl += ic ? 1 + bit : 0;
  }
}

// One warp per (code-block, bit-plane) item.
//
// 1. Column masks of the plane: significant before it (|q| >> (p+1) != 0),
//    magnitude bit p, refinement history (|q| >> (p+2) != 0), sign.
// 2. Significance propagation: the visited (V) and newly significant (N)
//    samples are the least fixpoint of the pass's visiting rule, iterated
//    over the whole block; each round also fills every newly significant
//    sample's run of magnitude-1 samples below it with one carry-propagating
//    addition, so only horizontal chains take extra rounds. The scan order
//    makes the rule causal, so the fixpoint is the sequential pass's result.
// 3. Cleanup masks, run-length columns and, bit-sliced, every sample's
//    symbols: zero-coding label with the neighbourhood of the pass that codes
//    it, refinement context, sign context and prediction bit.
// 4. Emission, stripe by stripe: each sample is coded in exactly one pass
//    (SP if visited, MR if significant before, else cleanup or a cleanup
//    run), so each lane writes its two columns' symbols into the three
//    streams (SP | MR | cleanup, whose starts are known from the totals) at
//    offsets from two packed warp scans.
__global__ void __launch_bounds__(kModelWarps * 32, 5) t1_model_kernel(T1Args a, T1Part part) {
  __shared__ ModelSmem sm_all[kModelWarps];
  const int lane = threadIdx.x & 31;
  const int wid = threadIdx.x >> 5;
  ModelSmem& sm = sm_all[wid];
  const uint32_t nwarps = gridDim.x * kModelWarps;
  const int xa = lane, xb = lane + 32;

  const uint32_t p0 = part < kT1Parts ? part : kT1Part0;
  const uint32_t count = a.counts[part == kT1Again ? kCountAgainItems : kCountItems + p0];
  const uint32_t from = part == kT1Again ? a.counts[kCountItems] : p0 * a.nitems;
  for (uint32_t i = blockIdx.x * kModelWarps + wid; i < count; i += nwarps) {
    const uint32_t blkno = a.items[from + i] >> 6;
    const BlockDesc d = a.blocks[blkno];
    const int w = d.w, h = d.h;
    const int mbp = a.res[blkno].mbp;
    const int j = (int)(a.items[from + i] & 63u);
    const uint32_t item = a.plane_base[blkno] + (uint32_t)j;
    const int p = mbp - 1 - j;
    const bool top = j == 0;
    const uint64_t rows = h >= 64 ? ~0ull : ((1ull << h) - 1);
    const uint64_t vA = xa < w ? rows : 0, vB = xb < w ? rows : 0;

    // ---- 1. column masks (made by t1_planes_kernel) ----
    auto ld = [&](const uint32_t* v, size_t row0, int x) {
      return (uint64_t)v[row0 + x] | (uint64_t)v[row0 + 64 + x] << 32;
    };
    const size_t pi = (size_t)item * 256;
    const uint64_t SA = ld(a.planes, pi, xa), SB = ld(a.planes, pi, xb);
    const uint64_t BA = ld(a.planes, pi + 128, xa), BB = ld(a.planes, pi + 128, xb);
    const uint64_t RA = top ? 0 : ld(a.planes, pi - 256, xa), RB = top ? 0 : ld(a.planes, pi - 256, xb);
    const uint64_t GA = ld(a.signs, (size_t)blkno * 128, xa), GB = ld(a.signs, (size_t)blkno * 128, xb);
    const Side sS = sides(SA, SB, lane);

    // ---- 2. significance propagation ----
    uint64_t NA = 0, NB = 0, VA = 0, VB = 0;
    if (!top) {
      // parts of the visiting rule on states before the pass: S below, E,
      // SE, NE (rows 1-3 of a stripe), SW (row 3)
      const uint64_t invA = (SA >> 1) | sS.ea | (sS.ea >> 1) | ((sS.ea << 1) & ~kRow0) | ((sS.wa >> 1) & kRow3);
      const uint64_t invB = (SB >> 1) | sS.eb | (sS.eb >> 1) | ((sS.eb << 1) & ~kRow0) | ((sS.wb >> 1) & kRow3);
      const uint64_t MA = BA & ~SA & vA, MB = BB & ~SB & vB;  // samples that turn significant when visited
      for (;;) {  // N grows every round until it is stable: at most 4096 rounds
        const uint64_t FA = SA | NA, FB = SB | NB;
        const Side f = sides(FA, FB, lane);
        VA = (invA | (FA << 1) | f.wa | (f.wa << 1) | ((f.wa >> 1) & ~kRow3) | ((f.ea << 1) & kRow0)) & ~SA & vA;
        VB = (invB | (FB << 1) | f.wb | (f.wb << 1) | ((f.wb >> 1) & ~kRow3) | ((f.eb << 1) & kRow0)) & ~SB & vB;
        uint64_t nA = VA & BA, nB = VB & BB;
        nA |= MA & ~(MA + nA);  // the run of M below each new sample
        nB |= MB & ~(MB + nB);
        const bool changed = nA != NA || nB != NB;
        NA = nA;
        NB = nB;
        if (!__any_sync(~0u, changed)) break;
      }
    }

    // ---- 3. cleanup masks and the symbol planes ----
    const uint64_t SNA = SA | NA, SNB = SB | NB;                // after SP
    const uint64_t CA = ~SNA & ~VA & vA, CB = ~SNB & ~VB & vB;  // coded in cleanup
    const uint64_t QA = CA & BA, QB = CB & BB;                  // significant in cleanup
    const uint64_t FA = SNA | QA, FB = SNB | QB;                // after cleanup
    const Side sSN = sides(SNA, SNB, lane), sF = sides(FA, FB, lane), sG = sides(GA, GB, lane);
    uint32_t ns_sp = __popcll(NA) + __popcll(NB), ns_cl = __popcll(QA) + __popcll(QB);
    uint32_t n_sp = __popcll(VA) + __popcll(VB) + ns_sp, sig_before = __popcll(SA) + __popcll(SB);
    #pragma unroll
    for (int col = 0; col < 2; ++col) {
      const uint64_t S = col ? SB : SA, B = col ? BB : BA, R = col ? RB : RA, G = col ? GB : GA;
      const uint64_t V = col ? VB : VA, SN = col ? SNB : SNA, C = col ? CB : CA, F = col ? FB : FA;
      const uint64_t valid = col ? vB : vA;
      const uint64_t Sw = col ? sS.wb : sS.wa, Se = col ? sS.eb : sS.ea;
      const uint64_t SNw = col ? sSN.wb : sSN.wa, SNe = col ? sSN.eb : sSN.ea;
      const uint64_t Fw = col ? sF.wb : sF.wa, Fe = col ? sF.eb : sF.ea;
      const uint64_t Gw = col ? sG.wb : sG.wa, Ge = col ? sG.eb : sG.ea;
      // cleanup runs (flags.rs:219-235): a full stripe of the column with
      // nothing significant or visited in it or around it (west column and
      // row above after cleanup, east column and row below before it)
      const uint64_t T = SN | V | Fw | SNe | (((Fw | F | Fe) << 1) & kRow0) | (((SNw | SN | SNe) >> 1) & kRow3);
      const uint64_t busy = (T | (T >> 1) | (T >> 2) | (T >> 3)) & kRow0;
      const uint64_t clean = ~busy & kRow0 & (valid >> 3);
      // neighbourhood at coding time: SP samples see the SP frames, the
      // others the cleanup frames
      const Hood hs = hood(SN, S, SNw, Sw, SNe, Se);
      const Hood hc = hood(F, SN, Fw, SNw, Fe, SNe);
      Hood hd;
      hd.nw = pick(V, hs.nw, hc.nw);
      hd.n = pick(V, hs.n, hc.n);
      hd.ne = pick(V, hs.ne, hc.ne);
      hd.w = pick(V, hs.w, hc.w);
      hd.e = pick(V, hs.e, hc.e);
      hd.sw = pick(V, hs.sw, hc.sw);
      hd.s = pick(V, hs.s, hc.s);
      hd.se = pick(V, hs.se, hc.se);
      uint64_t l[4], m[3], x;
      zc_label_planes(hd.nw, hd.n, hd.ne, hd.w, hd.e, hd.sw, hd.s, hd.se, (int)d.orient, l);
      sign_planes(hd.n, hd.s, hd.w, hd.e, G << 1, G >> 1, Gw, Ge, m, &x);
      // refinement context (helpers.rs:36-50): 16 after a first refinement,
      // else 15 with a significant neighbour (state after SP), else 14
      const uint64_t nb = (SN << 1) | (SN >> 1) | SNw | (SNw << 1) | (SNw >> 1) | SNe | (SNe << 1) | (SNe >> 1);
      const uint64_t mr1 = S & ~R;  // contexts 14 and 15: binary 0111x
      uint64_t out[kNumPlanes];
      out[kPlV] = V;
      out[kPlS] = S;
      out[kPlC] = C;
      out[kPlB] = B;
      out[kPlClean] = clean;
      out[kPlP0] = pick(S, mr1 & nb, l[0]);
      out[kPlP1] = pick(S, mr1, l[1]);
      out[kPlP2] = pick(S, mr1, l[2]);
      out[kPlP3] = pick(S, mr1, l[3]);
      out[kPlP4] = S & R;
      out[kPlM0] = m[0];
      out[kPlM1] = m[1];
      out[kPlM2] = m[2];
      out[kPlX] = x ^ G;
      const int xc = col ? xb : xa;
      #pragma unroll
      for (int k = 0; k < kNumPlanes; ++k) {
        sm.pl[k][0][xc] = (uint32_t)out[k];
        sm.pl[k][1][xc] = (uint32_t)(out[k] >> 32);
      }
    }
    n_sp = __reduce_add_sync(~0u, n_sp);
    sig_before = __reduce_add_sync(~0u, sig_before);
    ns_sp = __reduce_add_sync(~0u, ns_sp);
    ns_cl = __reduce_add_sync(~0u, ns_cl);
    __syncwarp();

    // ---- 4. emission, stripe by stripe ----
    uint8_t* out = a.sym + (size_t)item * a.sym_slot;
    const uint32_t at_mr = pad16(n_sp), at_cl = at_mr + pad16(sig_before);
    uint32_t pos_sp = 0, pos_mr = at_mr, pos_cl = at_cl;
    const int nstripes = (h + 3) >> 2;
    for (int half = 0; half < 2 && 8 * half < nstripes; ++half) {
      uint32_t qa[kNumPlanes], qb[kNumPlanes];
      #pragma unroll
      for (int k = 0; k < kNumPlanes; ++k) {
        qa[k] = sm.pl[k][half][xa];
        qb[k] = sm.pl[k][half][xb];
      }
      const int send = min(8, nstripes - 8 * half);
      for (int s = 0; s < send; ++s) {
        const uint32_t vA4 = nib(qa[kPlV], s), sA4 = nib(qa[kPlS], s), cA4 = nib(qa[kPlC], s),
                       bA4 = nib(qa[kPlB], s), lA = nib(qa[kPlClean], s) & 1u;
        const uint32_t vB4 = nib(qb[kPlV], s), sB4 = nib(qb[kPlS], s), cB4 = nib(qb[kPlC], s),
                       bB4 = nib(qb[kPlB], s), lB = nib(qb[kPlClean], s) & 1u;
        uint32_t totA, totB;
        const uint32_t offA = warp_offset(column_counts(vA4, sA4, cA4, bA4, lA), lane, &totA);
        const uint32_t offB = warp_offset(column_counts(vB4, sB4, cB4, bB4, lB), lane, &totB);
        // primary and sign symbols of the 4 rows, one per byte
        uint32_t primA = spread4(bA4) << 7, primB = spread4(bB4) << 7;
        #pragma unroll
        for (int k = 0; k < 5; ++k) {
          primA |= spread4(nib(qa[kPlP0 + k], s)) << k;
          primB |= spread4(nib(qb[kPlP0 + k], s)) << k;
        }
        uint32_t sgnA = 0x08080808u | spread4(nib(qa[kPlX], s)) << 7, sgnB = 0x08080808u | spread4(nib(qb[kPlX], s)) << 7;
        #pragma unroll
        for (int k = 0; k < 3; ++k) {
          sgnA |= spread4(nib(qa[kPlM0 + k], s)) << k;
          sgnB |= spread4(nib(qb[kPlM0 + k], s)) << k;
        }
        uint8_t* osp = out + pos_sp + (offA & 0x7ffu);
        uint8_t* omr = out + pos_mr + ((offA >> 11) & 0x3ffu);
        uint8_t* ocl = out + pos_cl + (offA >> 21);
        emit_column(vA4, sA4, cA4, bA4, lA, primA, sgnA, osp, omr, ocl);
        osp = out + pos_sp + (totA & 0x7ffu) + (offB & 0x7ffu);
        omr = out + pos_mr + ((totA >> 11) & 0x3ffu) + ((offB >> 11) & 0x3ffu);
        ocl = out + pos_cl + (totA >> 21) + (offB >> 21);
        emit_column(vB4, sB4, cB4, bB4, lB, primB, sgnB, osp, omr, ocl);
        pos_sp += (totA & 0x7ffu) + (totB & 0x7ffu);
        pos_mr += ((totA >> 11) & 0x3ffu) + ((totB >> 11) & 0x3ffu);
        pos_cl += (totA >> 21) + (totB >> 21);
      }
    }
    // padding of each pass to whole 16-symbol chunks
    if (pos_sp + lane < at_mr) out[pos_sp + lane] = (uint8_t)kPadSymbol;
    if (pos_mr + lane < at_cl) out[pos_mr + lane] = (uint8_t)kPadSymbol;
    if (pos_cl + lane < pad16(pos_cl)) out[pos_cl + lane] = (uint8_t)kPadSymbol;
    if (lane == 0) {
      ItemRec rec;
      rec.n_sp = n_sp;
      rec.n_mr = sig_before;
      rec.n_cl = pos_cl - at_cl;
      rec.ns_sp = ns_sp;
      rec.ns_cl = ns_cl;
      rec.sig_before = sig_before;
      rec.bitplane = (uint32_t)p;
      rec.remain = a.item_rec[item].remain;
      a.item_rec[item] = rec;
    }
    __syncwarp();
  }
}

// --------------------------------------------------------------------- MQ --
// The coder runs one code-block per lane, 1 to 32 lanes of a warp. A symbol
// takes the same instructions on every lane whatever it does, so a warp of 32
// blocks issues as many as a warp of one. What bounds it: in batches the
// ALU pipe (half rate; 77 % busy) and the latency of the context entries in
// shared memory; on a single page one chain's latency.
//
// - Interval register as a float in [1, 2) (A / 2^15): A - Qe, its comparison
//   with Qe and the renormalised result are exact in 24 bits, and
//   renormalisation is a logic operation that sets the exponent, where an
//   integer needs a leading-zero count and a shift on the chain.
// - The code register and the byte output, which part the lanes of a warp
//   when done per symbol, are done once per 16 symbols (mq_chunk16).
// - Each pass's symbols are padded to whole 16-symbol chunks with symbols that
//   change nothing (t1_model_kernel), so a pass ends between two chunks.
//
// Measured with every pass coded (2550x3300 gray q85 page; batch of 24 sRGB q75
// pages): 3.04 and 5.2 ms; 4.38 and 11.1 ms with an integer coder split over two
// warps on the page and branching at its byte output in the batch. Now that
// blocks stop early the page's takes 1.6 ms. A lone chain takes 90 cycles per
// symbol (32 lanes and 16 warps per SM: 490 G symbols/s); 106 when predicates
// chose between A and Qe, and a renormalised context's state was read only then.
//
// Context entry, in shared memory: x = Qe / 2^15 as a float, its sign bit the
// MPS; y = shared address of the state's successors in the table | MPS << 3. The
// table holds per state (state, MPS pair) its successors' entries: after an MPS
// renormalisation, then after an LPS.
struct __align__(16) MqTable {
  uint2 next[kStates][2];
};
// Entry of a state; `table` is the table's shared address. kNoState: padding,
// whose Qe of 0 changes nothing.
constexpr uint32_t kNoState = kStates;
__device__ __forceinline__ uint2 mq_entry(uint32_t state, uint32_t table) {
  if (state == kNoState) return make_uint2(0u, table);
  const uint32_t qe = c_mq[state] & 0xffffu, mps = state & 1u;
  return make_uint2(__float_as_uint((float)qe * (1.0f / 32768.0f)) | mps << 31, (table + state * 16u) | mps << 3);
}
__device__ __forceinline__ uint32_t mq_state(uint2 e, uint32_t table) { return (e.y - table) >> 4; }
__device__ __forceinline__ uint32_t mq_table_at(const MqTable& t) {
  return (uint32_t)__cvta_generic_to_shared(&t);
}
__device__ __forceinline__ void load_mq_table(MqTable& t) {
  const uint32_t at = mq_table_at(t);
  for (uint32_t i = threadIdx.x; i < kStates; i += blockDim.x) {
    const uint32_t v = c_mq[i];
    t.next[i][0] = mq_entry((v >> 16) & 0xffu, at);
    t.next[i][1] = mq_entry(v >> 24, at);
  }
}

struct Mq {
  float a;        // interval, A / 2^15 in [1, 2)
  uint32_t c;     // code register
  int ct;         // shifts left until a byte is cut
  uint32_t last;  // the last byte cut, before the next one's carry into it
  uint8_t* at;    // its place; a block's slot begins with the pre-byte
};

// Payload bytes are written by volatile assembly, which keeps its order: a
// byte may be written again by mq_shift.
__device__ __forceinline__ void put_byte(uint8_t* at, uint32_t v) {
  asm volatile("st.global.u8 [%0], %1;" ::"l"(at), "r"(v));
}

// Adds to the code register and shifts it by n bits, cutting bytes as it
// fills (BYTEOUT, src/mq/mod.rs:382-404).
__device__ __forceinline__ void mq_shift(Mq& m, uint32_t add, int n) {
  uint32_t c = m.c + add;
  while (n >= m.ct) {
    c <<= m.ct;
    n -= m.ct;
    if (m.last != 0xffu && (c & 0x8000000u) != 0) {
      ++m.last;
      if (m.last == 0xffu) c &= 0x7ffffffu;
    }
    put_byte(m.at++, m.last);
    const bool big = m.last == 0xffu;
    m.last = (big ? c >> 20 : c >> 19) & 0xffu;
    c &= big ? 0xfffffu : 0x7ffffu;
    m.ct = big ? 7 : 8;
  }
  m.ct -= n;
  m.c = c << n;
}

// Context entries of a CTA's lanes: context c of thread t at byte
// c * kCtxStride + 8 t (no bank conflicts whatever contexts the lanes use).
constexpr uint32_t kCtxStride = kMqWarps * 32 * 8;
static_assert(kCtxStride == 1024, "the context offset is a shift of the symbol");
struct MqSmem {
  __align__(16) uint8_t ce[kMqCtx * kCtxStride];
  MqTable table;
};
__device__ __forceinline__ uint2& ctx_at(MqSmem& sm, uint32_t off) {
  return *reinterpret_cast<uint2*>(sm.ce + off);
}
// Offset of the context entry of symbol i (0..3) of a word for the lane whose
// entries start at `lane`; the symbol's decision as a sign bit; and as bit 3.
__device__ __forceinline__ uint32_t sym_ctx(uint32_t w, int i, uint32_t lane) {
  return ((i < 2 ? w << (10 - 8 * i) : w >> (8 * i - 10)) & 0x7c00u) | lane;
}
__device__ __forceinline__ uint32_t sym_sign(uint32_t w, int i) { return w << (24 - 8 * i); }
__device__ __forceinline__ uint32_t sym_bit3(uint32_t w, int i) { return (w >> (8 * i + 4)) & 8u; }

// Codes the 16 symbols of a chunk.
//
// A symbol (C.2.4-C.2.7) with the decisions folded: after A -= Qe the coder
// keeps A (and adds Qe to C) exactly when (A < Qe) equals "LPS", and
// otherwise takes Qe (C unchanged): of the two the larger for an MPS, the
// smaller for an LPS, which with both negative is the larger again (predicates
// would cost the chain more than signs). The context moves to its next state
// exactly when the result is below 0x8000 and is renormalised.
//
// The code register is brought up to date once for the chunk: its 16
// additions are summed at 31 fractional bits (`acc`), each at the shift it
// comes at, and bytes are cut from the sum. A byte is then cut with additions
// in the sum that come after it. They can only carry one into it, as the
// next cut would have found; what they could get wrong is a byte of 0xFF
// that such a carry turns to zeros, so a byte of zeros with the three bits
// below it zero too (a carry adds less than their weight) makes the chunk
// take the additions one by one, as does one that shifts by more than 31
// bits.
__device__ __forceinline__ void mq_chunk16(Mq& m, MqSmem& sm, uint32_t lane, const uint4 q) {
  const uint32_t w[5] = {q.x, q.y, q.z, q.w, kPadSymbol};
  uint32_t ops[16];  // exponent of the result (127 - the shift) << 23 | addition to C
  uint64_t acc = 0;
  int room = 31;  // fractional bits left: 31 - shifts so far
  uint32_t cx = sym_ctx(w[0], 0, lane);
  uint2 e = ctx_at(sm, cx);
  #pragma unroll
  for (int i = 0; i < 16; ++i) {
    const uint32_t cxn = sym_ctx(w[(i + 1) >> 2], (i + 1) & 3, lane);
    const uint2 en = ctx_at(sm, cxn);  // the next symbol's entry, one step ahead
    const uint32_t next = e.y ^ sym_bit3(w[i >> 2], i & 3);
    uint2 s;  // the state it may move to, read while A is found
    asm("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(s.x), "=r"(s.y) : "r"(next));
    const uint32_t xs = e.x ^ (sym_sign(w[i >> 2], i & 3) & 0x80000000u);
    const float a = __fsub_rn(m.a, fabsf(__uint_as_float(e.x)));
    const float sa = __uint_as_float(__float_as_uint(a) | (xs & 0x80000000u)), sq = __uint_as_float(xs);
    const float v = fmaxf(sa, sq);
    // sa >= sq for an MPS, > for an LPS: both are multiples of 2^-15
    const bool take_a = sa > __fmul_rn(sq, 1.0f - 1.0f / 1048576.0f);
    const uint32_t vb = __float_as_uint(v);
    m.a = __uint_as_float((vb & 0x7fffffu) | 0x3f800000u);
    // at 256 a unit of the last place is 2^-15
    const uint32_t add = __float_as_uint(__fadd_rn(take_a ? fabsf(sq) : 0.0f, 256.0f)) & 0xffffu;
    ops[i] = (vb & 0x7f800000u) | add;
    acc += (uint64_t)add * __funnelshift_l(0u, 1u, (uint32_t)room);
    room += (int)(ops[i] >> 23) - 127;
    const bool renormalised = fabsf(v) < 1.0f;
    if (renormalised) ctx_at(sm, cx) = s;
    const bool same = renormalised && cxn == cx;
    e.x = same ? s.x : en.x;
    e.y = same ? s.y : en.y;
    cx = cxn;
  }
  bool one_by_one = room < 0;
  if (!one_by_one) {
    uint64_t x = (((uint64_t)m.c << 31) + acc) << m.ct;  // C at its next cut, 31 fractional bits
    int t = m.ct + room - 31;                            // shifts that cut lacks
    uint32_t last = m.last;
    uint8_t* at = m.at;
    while (t <= 0) {
      const uint32_t hi = (uint32_t)(x >> 32);  // C's bit k at k - 1
      one_by_one |= ((hi >> 15) & 0x7ffu) == 0;
      const uint32_t done = last == 0xffu ? 0xffu : last + (hi >> 26);  // with the carry
      const bool big = done == 0xffu;
      put_byte(at++, done);
      // after 0xFF a byte takes 7 bits, and the carry place when it was
      // 0xFF before the carry
      last = big ? (last == 0xffu ? hi >> 19 : (hi >> 19) & 0x7fu) : (hi >> 18) & 0xffu;
      const int bits = big ? 7 : 8;
      x = ((uint64_t)(hi & (big ? 0x7ffffu : 0x3ffffu)) << 32 | (uint32_t)x) << bits;
      t += bits;
    }
    if (!one_by_one) {
      m.c = (uint32_t)(x >> 32) >> (t - 1);
      m.ct = t;
      m.last = last;
      m.at = at;
    }
  }
  if (one_by_one) {
    // (rolled: unrolled sixteen times it took the registers of the code above)
    #pragma unroll 1
    for (int h = 0; h < 4; ++h) {
      #pragma unroll
      for (int i = 0; i < 4; ++i) mq_shift(m, ops[i] & 0xffffu, 127 - (int)(ops[i] >> 23));
      #pragma unroll
      for (int i = 0; i < 12; ++i) ops[i] = ops[i + 4];
    }
  }
}

// Stopping a block's coding once rate control can no longer choose any of its
// later passes. Rate control keeps, of a block's passes, the one that
// maximises (distortion removed - lambda * bytes). `lead` is how far the best
// pass so far lies above the last one in that measure; a later pass can add at
// most ItemRec::remain to the last one's distortion and never takes bytes
// back, so once remain < lead none of them is chosen. The chosen pass's bytes
// are then final too: lead > 0 means that bytes were cut after them, and a
// byte is final once the next one is cut.
//
// lambda is lambda_raw unless the component's largest slope is small, and
// then in proportion to that slope. So a block may only stop once some block
// of its component (not necessarily this one) has shown a slope that settles
// lambda, or a half, a quarter or an eighth as large: lambda is then at least
// that share of lambda_raw, and the block, measured with it, may stop unless a
// later pass could still raise the largest slope. A block that has not been
// stopped gives its largest slope as before. A block's last pass shows no
// slope: it takes the termination's bytes too, which are not in its count yet.
//
// The sums are f32: `slack` bounds their rounding against the f64 curve (a
// term is within 1e-6 of its value, and each of at most 124 passes adds two
// roundings of the lead).
// On a 2550x3300 gray q85 page 33 % of the symbols are coded, and 37 k of the
// longest block's 58 k.
constexpr int kLevels = 4;
struct StopState {
  float lead[kLevels];  // with lambda_raw, a half, a quarter, an eighth of it
  float slack, total;
  uint32_t prev;  // bytes after the last pass (a header of 2 counts to the first one)
};
struct Stop {
  float unit, lambda, slope;
  StopState s;
  uint32_t* flag;  // [k]: a slope of 2^-k times the one that settles lambda was seen
  __device__ __forceinline__ void start(const T1Args& a, uint32_t b, const BlockDesc& d) {
    const CompParam& cp = a.comps[d.comp_key];
    unit = block_unit(a, b, d);
    lambda = cp.lambda;
    slope = cp.settled;
    flag = a.settled + kLevels * d.comp_key;
    s = StopState{};
    s.prev = 0u - 2u;
  }
  __device__ __forceinline__ bool seen(int k) const { return reinterpret_cast<const volatile uint32_t*>(flag)[k] != 0u; }
  __device__ __forceinline__ void pass(uint32_t pos, float samples, int bitplane) {
    if (!flag) return;
    const float gain = samples * unit * plane_energy(bitplane);
    float cost = lambda * (float)(pos - s.prev);
    s.slack += 2e-5f * (gain + cost);
    s.total += gain;
    s.prev = pos;
    float need = slope * (float)(pos + 2u);
    #pragma unroll
    for (int k = 0; k < kLevels; ++k) {
      s.lead[k] = fmaxf(0.0f, s.lead[k] - gain + cost);
      if (s.total * 0.9999f >= need) reinterpret_cast<volatile uint32_t*>(flag)[k] = 1u;
      cost *= k == 0 ? 0.49999f : 0.5f;
      need *= 0.5f;
    }
  }
  __device__ __forceinline__ bool here(float remain) const {
    if (!flag) return false;
    const float most = (s.total + remain) * 1.0001f;  // over bytes: the largest slope a later pass can give
    float shown = slope * (float)(s.prev + 2u);
    #pragma unroll
    for (int k = 0; k < kLevels; ++k, shown *= 0.5f)
      if (remain + s.slack < s.lead[k] && (k == 0 || most < shown) && seen(k)) return true;
    return false;
  }
};

// What a block's coding goes on from in the second round, at the end of its
// payload slot (which no block of pixels comes near).
struct MqState {
  Mq m;
  StopState stop;
  uint16_t context[kMqCtx];
};
constexpr uint32_t kStateBytes = 144;
static_assert(sizeof(MqState) <= kStateBytes && kCtxNone <= kMqCtx, "the slot's end");

// MQ-codes code-block b on the calling lane, or nothing when b is kNoBlock;
// every lane of the warp calls. The lanes meet at every chunk (the vote):
// left to themselves, a lane that ends a pass falls behind the others and
// each would run the chunk code on its own.
constexpr uint32_t kNoBlock = 0xffffffffu;
template <int round>
__device__ __forceinline__ void mq_code_block(const T1Args& a, uint32_t b, MqSmem& sm) {
  const uint32_t lane = threadIdx.x * 8u, table = mq_table_at(sm.table);
  BlockOut o{};
  if (b != kNoBlock) o = a.res[b];
  const int mbp = o.status ? 0 : o.mbp;
  bool active = mbp > 0;
  BlockDesc d{};
  uint32_t base = 0;
  int j = 0, modelled = 0;  // item; those of the round end before this one
  ItemRec r{};
  const uint4* src = nullptr;
  uint4 c0 = make_uint4(0u, 0u, 0u, 0u);
  if (active) {
    d = a.blocks[b];
    modelled = round ? mbp : (int)a.nplanes[b];
    j = round ? (int)a.nplanes[b] : 0;
    base = a.plane_base[b];
    r = a.item_rec[base + j];
    src = reinterpret_cast<const uint4*>(a.sym + (size_t)(base + j) * a.sym_slot);
    c0 = src[0];  // the slot and buffer are padded for these reads
    // contexts: state 0 except UNI 46, AGG 3, ZC 4 (src/mq/mod.rs:195-200)
    for (uint32_t c = 0; c < kMqCtx; ++c)
      ctx_at(sm, c * kCtxStride + lane) =
          mq_entry(c == kCtxNone ? kNoState : c == kCtxUNI ? 92 : c == kCtxAGG ? 6 : c == 0 ? 8 : 0, table);
  }
  Stop stop{};
  if (active && a.settled && !a.comps[d.comp_key].lossless) stop.start(a, b, d);
  uint8_t* const slot = a.out + d.out_off;
  MqState* const state = reinterpret_cast<MqState*>(slot + d.out_cap - kStateBytes);
  const uint8_t* const slot_end = slot + d.out_cap - kStateBytes - 40;  // a chunk cuts at most 35 bytes
  Mq m{1.0f, 0u, 12, 0u, slot};
  bool ovf = false;
  PassRec* pr = a.passes + d.pass_off;
  if (round && active) {
    m = state->m;
    stop.s = state->stop;
    for (uint32_t c = 0; c < kCtxNone; ++c) ctx_at(sm, c * kCtxStride + lane) = mq_entry(state->context[c], table);
    pr += 1 + 3 * (j - 1);
  }
  // One flat loop over the chunks of all items (bit-planes); the next item's
  // record and first chunk are fetched during the current item's last chunk.
  ItemRec rn = r;
  uint4 n0 = c0;
  uint32_t nsym = 0, left = 0, ahead = 0;  // symbols; chunks of the pass and of the item
  int k = 0;                               // pass: SP, MR, cleanup (the first item has only its cleanup)
  auto record = [&] {                   // numbytes() after the pass
    const uint32_t pos = (uint32_t)(m.at - slot);
    const uint8_t bp = (uint8_t)r.bitplane;
    if (k == 2)
      *pr = PassRec{pos, r.ns_cl, j == 0 ? 0u : r.sig_before + r.ns_sp, 2, bp, 0};
    else if (k == 0)
      *pr = PassRec{pos, r.ns_sp, r.sig_before, 0, bp, 0};
    else
      *pr = PassRec{pos, 0u, r.sig_before, 1, bp, 0};
    ++pr;
    if (k == 2 && j + 1 == mbp) return;  // the last pass: its bytes are known only after termination
    stop.pass(pos, k == 2 ? 0.85f * (float)r.ns_cl : (k == 0 ? (float)r.ns_sp : 0.25f * (float)r.sig_before), bp);
  };
  // the first pass of item j that has symbols
  auto start_item = [&] {
    nsym += r.n_sp + r.n_mr + r.n_cl;
    ahead = ((r.n_sp + 15u) >> 4) + ((r.n_mr + 15u) >> 4) + ((r.n_cl + 15u) >> 4);
    k = j == 0 ? 2 : 0;
    left = ((j == 0 ? r.n_cl : r.n_sp) + 15u) >> 4;
    while (k < 2 && left == 0) {
      record();
      ++k;
      left = ((k == 1 ? r.n_mr : r.n_cl) + 15u) >> 4;
    }
  };
  if (active) start_item();
  bool stopped = false, unfinished = false;
  while (__any_sync(0xffffffffu, active)) {
    if (!active) continue;
    if (ahead == 1 && j + 1 < modelled) {
      rn = a.item_rec[base + j + 1];
      const uint4* ns = reinterpret_cast<const uint4*>(a.sym + (size_t)(base + j + 1) * a.sym_slot);
      n0 = ns[0];
    }
    const uint4 q = c0;
    c0 = src[1];  // 16 bytes ahead: inside the slot or the buffer's pad
    ++src;
    mq_chunk16(m, sm, lane, q);
    if (m.at > slot_end) {  // no room for another chunk: the block has failed
      ovf = true;
      m.at = slot;
    }
    --ahead;
    if (--left == 0) {
      record();
      while (k < 2 && left == 0) {  // the next pass that has symbols
        ++k;
        left = ((k == 1 ? r.n_mr : r.n_cl) + 15u) >> 4;
        if (left == 0) record();
      }
      if (left == 0) {  // the next item
        stopped = j + 1 < mbp && stop.here(r.remain);
        ++j;
        unfinished = !stopped && j == modelled && j < mbp;
        if (stopped || j == modelled) {
          active = false;
        } else {
          r = rn;
          src = reinterpret_cast<const uint4*>(a.sym + (size_t)(base + j) * a.sym_slot);
          c0 = n0;
          start_item();
        }
      }
    }
  }
  if (mbp == 0) return;
  atomicAdd(a.sym_count, (unsigned long long)nsym);
  if (unfinished && !ovf) {  // the second round goes on with the other bit-planes
    state->m = m;
    state->stop = stop.s;
    for (uint32_t c = 0; c < kCtxNone; ++c) state->context[c] = (uint16_t)mq_state(ctx_at(sm, c * kCtxStride + lane), table);
    a.unfinished[atomicAdd(a.counts + kCountUnfinished, 1u)] = b;
    return;
  }
  if (stopped || unfinished) {  // the coded passes stand, each with its bytes so far
    o.npasses = (uint16_t)(1 + 3 * (j - 1));
    o.payload_len = (uint32_t)(m.at - slot);
    o.status = ovf ? 1 : 0;
    a.res[b] = o;
    return;
  }
  // termination (src/mq/mod.rs:244-250, 373-379)
  uint32_t c = m.c;
  const uint32_t t = c + ((__float_as_uint(m.a) & 0x7fffffu) | 0x800000u) / 256u;
  c |= 0xffffu;
  if (c >= t) c -= 0x8000u;
  m.c = c;
  mq_shift(m, 0u, m.ct);
  mq_shift(m, 0u, m.ct);
  put_byte(m.at, m.last);
  const uint32_t pos = (uint32_t)(m.at - slot);
  o.payload_len = m.last == 0xffu ? pos - 1 : pos;  // take_bytes
  o.status = ovf ? 1 : 0;
  a.res[b] = o;
}

// As few blocks per warp as keep at most one warp on each of the SMs' four
// schedulers (a warp's lanes cost nothing, and a second warp on a scheduler
// lengthens both warps' chains), up to 32.
JP2G_HD int mq_blocks_auto(uint32_t nblocks, uint32_t warps) {
  const uint32_t n = (nblocks + warps - 1) / warps;
  return n < 1u ? 1 : n > 32u ? 32 : (int)n;
}

// The part's first block in the order.
__device__ __forceinline__ uint32_t part_first(const T1Args& a, T1Part part) {
  return part == kT1Part1 ? a.counts[kCountBlocks] : 0u;
}

// Warp w codes blocks order[w * bpw + lane], lanes < bpw. bpw 0: automatic
// for `warps` warps.
// (Four CTAs fit an SM. Asked for three, the compiler orders a chunk's work with
// three registers more and a chain takes 3 % less.)
template <int round>
__global__ void __launch_bounds__(kMqWarps * 32, 3) t1_mq_kernel(T1Args a, T1Part part, int bpw, uint32_t warps) {
  __shared__ MqSmem sm;
  load_mq_table(sm.table);
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int wid = threadIdx.x >> 5;
  if constexpr (round == 0) {
    const uint32_t n = part == kT1All ? a.nblocks : a.counts[kCountBlocks + part];
    const uint32_t first = part_first(a, part);
    if (bpw == 0) bpw = mq_blocks_auto(n, warps);
    const uint32_t slot = (blockIdx.x * kMqWarps + wid) * (uint32_t)bpw + (uint32_t)lane;
    mq_code_block<0>(a, lane < bpw && slot < n ? a.mq_order[first + slot] : kNoBlock, sm);
  } else {  // the blocks that t1_recheck_kernel listed, over a fixed grid
    const uint32_t count = a.counts[kCountAgainBlocks];
    if (bpw == 0) bpw = mq_blocks_auto(count, warps);
    const uint32_t per_cta = kMqWarps * (uint32_t)bpw;
    for (uint32_t first = blockIdx.x * per_cta; first < count; first += gridDim.x * per_cta) {
      const uint32_t slot = first + (uint32_t)(wid * bpw + lane);
      mq_code_block<1>(a, lane < bpw && slot < count ? a.again[slot] : kNoBlock, sm);
    }
  }
}

// Between the rounds: of the blocks left unfinished, those that may stop
// where they are (their component's lambda was not settled when they got
// there) are done; the others are listed for the second round with their
// remaining items.
__global__ void t1_recheck_kernel(T1Args a) {
  const uint32_t count = a.counts[kCountUnfinished];
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
    const uint32_t b = a.unfinished[i];
    const BlockDesc d = a.blocks[b];
    BlockOut o = a.res[b];
    uint8_t* const slot = a.out + d.out_off;
    const MqState& state = *reinterpret_cast<const MqState*>(slot + d.out_cap - kStateBytes);
    const uint32_t done = a.nplanes[b], all = o.mbp;
    Stop stop;
    stop.start(a, b, d);
    stop.s = state.stop;
    if (stop.here(a.item_rec[a.plane_base[b] + done - 1].remain)) {
      o.npasses = (uint16_t)(1 + 3 * (done - 1));
      o.payload_len = (uint32_t)(state.m.at - slot);
      a.res[b] = o;
      continue;
    }
    a.again[atomicAdd(a.counts + kCountAgainBlocks, 1u)] = b;
    const uint32_t at = a.counts[kCountItems] + atomicAdd(a.counts + kCountAgainItems, all - done);
    for (uint32_t j = done; j < all; ++j) a.items[at + j - done] = b << 6 | j;
  }
}

}  // namespace

// The bit-sliced context formation evaluated on single samples, in the
// layout of the context tables (jp2g_debug_context_labels).
void context_labels_from_logic(uint8_t* zc, uint8_t* sc, uint8_t* spb) {
  for (int o = 0; o < 4; ++o)
    for (uint32_t f = 0; f < 512; ++f) {
      uint32_t l[4];
      zc_label_planes<uint32_t>(f & 1u, (f >> 1) & 1u, (f >> 2) & 1u, (f >> 3) & 1u, (f >> 5) & 1u,
                                (f >> 6) & 1u, (f >> 7) & 1u, (f >> 8) & 1u, o, l);
      zc[o * 512 + f] = (uint8_t)((l[0] & 1u) | (l[1] & 1u) << 1 | (l[2] & 1u) << 2 | (l[3] & 1u) << 3);
    }
  // sign index: bit 3 W, 0 W negative, 1 N, 4 N negative, 5 E, 2 E negative, 7 S, 6 S negative
  for (uint32_t f = 0; f < 256; ++f) {
    uint32_t m[3], x;
    sign_planes<uint32_t>((f >> 1) & 1u, (f >> 7) & 1u, (f >> 3) & 1u, (f >> 5) & 1u, (f >> 4) & 1u, (f >> 6) & 1u,
                          f & 1u, (f >> 2) & 1u, m, &x);
    sc[f] = (uint8_t)(8u + ((m[0] & 1u) | (m[1] & 1u) << 1 | (m[2] & 1u) << 2));
    spb[f] = (uint8_t)(x & 1u);
  }
}

bool upload_t1_tables(const uint32_t* mq) { return cudaMemcpyToSymbol(c_mq, mq, sizeof c_mq) == cudaSuccess; }

void launch_t1_analyze(const T1Args& a, cudaStream_t st) {
  if (a.nblocks == 0) return;
  const uint32_t threads = 256;
  const uint32_t grid = (uint32_t)(((uint64_t)a.nblocks * 32 + threads - 1) / threads);
  t1_analyze_kernel<<<grid, threads, 0, st>>>(a);
}

void launch_t1_planes(const T1Args& a, cudaStream_t st) {
  if (a.nblocks == 0) return;
  t1_planes_kernel<<<(uint32_t)(((uint64_t)a.nblocks * 32 + 255) / 256), 256, 0, st>>>(a);
}

void launch_t1_split(const T1Args& a, cudaStream_t st) {
  if (a.nblocks == 0) return;
  t1_split_kernel<<<(a.nblocks + 255) / 256, 256, 0, st>>>(a);
}

// CTAs loop over the items. A split wave's are short, as the coding of an
// earlier part waits for their places. The second round's items are few on most
// pages (39 blocks' of 24 sRGB ones) and many where the content is regular, so
// it has as many CTAs as the SMs hold at once.
void launch_t1_model(const T1Args& a, int num_sms, T1Part part, cudaStream_t st) {
  if (a.nitems == 0) return;
  uint32_t need = (a.nitems + kModelWarps - 1) / kModelWarps;
  uint32_t cap = (uint32_t)num_sms * (part == kT1Again ? 5 : part == kT1All ? 6 * 4 : 6 * 24);
  t1_model_kernel<<<need < cap ? need : cap, kModelWarps * 32, 0, st>>>(a, part);
}

void launch_t1_mq(const T1Args& a, int num_sms, int bpw, T1Part part, cudaStream_t st) {
  if (a.nblocks == 0) return;
  const uint32_t sms = (uint32_t)num_sms;
  if (bpw < 1 || bpw > 32) bpw = 0;
  const uint32_t most = (uint32_t)(bpw ? bpw : mq_blocks_auto(a.nblocks, sms * 4u));
  if (part == kT1Again) {  // four CTAs fit an SM; the first ones take a short list
    t1_mq_kernel<1><<<sms * 4, kMqWarps * 32, 0, st>>>(a, part, bpw, sms * 4u);
    return;
  }
  // a part of the wave's blocks takes a CTA on each SM, or as many blocks per warp as the whole wave
  const uint32_t per_cta = most * kMqWarps, all = (a.nblocks + per_cta - 1) / per_cta;
  t1_mq_kernel<0><<<bpw ? all : std::max(all, sms), kMqWarps * 32, 0, st>>>(a, part, bpw, sms * 4u);
}

void launch_t1_recheck(const T1Args& a, int num_sms, cudaStream_t st) {
  t1_recheck_kernel<<<(uint32_t)num_sms, 128, 0, st>>>(a);
}

namespace {
constexpr uint32_t kOrderBuckets = kOrderScratch / 2;

// Bucket of a block: its MQ symbol count / 64, clamped, reversed so that
// bucket 0 holds the largest blocks, and the LL bands' (few, and the ones whose
// slopes settle their components' lambda).
__device__ __forceinline__ uint32_t order_bucket(const T1Args& a, uint32_t b) {
  if (a.blocks[b].orient == 0) return 0;
  const uint32_t i0 = a.plane_base[b], i1 = i0 + a.nplanes[b];
  uint32_t n = 0;
  for (uint32_t i = i0; i < i1; ++i) {
    const ItemRec r = a.item_rec[i];
    n += r.n_sp + r.n_mr + r.n_cl;
  }
  const uint32_t k = min(n >> 6, kOrderBuckets - 1);
  return kOrderBuckets - 1 - k;
}

__device__ __forceinline__ bool in_part(const T1Args& a, T1Part part, uint32_t b) {
  return part == kT1All || part_of(a, b) == part;
}

__global__ void order_hist_kernel(T1Args a, T1Part part, uint32_t* key, uint32_t* hist) {
  const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= a.nblocks || !in_part(a, part, b)) return;
  const uint32_t k = order_bucket(a, b);
  key[b] = k;
  atomicAdd(hist + k, 1u);
}

// One CTA of 1024 threads: exclusive scan of the bucket counts into cursors.
__global__ void order_scan_kernel(const uint32_t* hist, uint32_t* cursor) {
  __shared__ uint32_t warp_tot[32];
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
  const uint32_t v = hist[t];
  uint32_t x = v;
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) warp_tot[wid] = x;
  __syncthreads();
  if (wid == 0) {
    uint32_t y = warp_tot[lane];
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t z = __shfl_up_sync(0xffffffffu, y, o);
      if (lane >= o) y += z;
    }
    warp_tot[lane] = y;
  }
  __syncthreads();
  cursor[t] = x - v + (wid > 0 ? warp_tot[wid - 1] : 0u);
}

__global__ void order_scatter_kernel(T1Args a, T1Part part, const uint32_t* key, uint32_t* cursor, uint32_t* order) {
  const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= a.nblocks || !in_part(a, part, b)) return;
  order[part_first(a, part) + atomicAdd(cursor + key[b], 1u)] = b;
}
}  // namespace

void launch_mq_order(const T1Args& a, T1Part part, uint32_t* order, uint32_t* key, uint32_t* scratch, cudaStream_t st) {
  if (a.nblocks == 0) return;
  uint32_t* hist = scratch;
  uint32_t* cursor = scratch + kOrderBuckets;
  cudaMemsetAsync(hist, 0, kOrderBuckets * sizeof(uint32_t), st);
  const uint32_t g = (a.nblocks + 255) / 256;
  order_hist_kernel<<<g, 256, 0, st>>>(a, part, key, hist);
  order_scan_kernel<<<1, kOrderBuckets, 0, st>>>(hist, cursor);
  order_scatter_kernel<<<g, 256, 0, st>>>(a, part, key, cursor, order);
}

}  // namespace jp2g
