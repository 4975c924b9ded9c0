// Tier-1 decoding on the device: the MQ decoder and the three decoding
// passes of every code-block (decode_codeblock, src/decode/t1.rs:87-210;
// the MQ decoder of src/mq/mod.rs; the context rules of src/tier1/*).
//
// Decoding is sequential within a code-block (every decoded bit changes the
// contexts of the samples after it). A warp decodes a block, every lane in
// the same control flow, so that what a symbol needs is spread over the
// lanes' registers and reached by shuffles:
//  - lane L owns columns L and L + 32 of the block (64-bit masks, bit y =
//    row y: significant, sign, visited, refined) and prepares, for 32
//    columns of a stripe at once, which of their samples the pass may code
//    and from which neighbourhood;
//  - lane c < 19 holds context c of the coder and its state's successors;
//  - the interval and code registers are the same in all lanes.
// What remains per symbol is one chain: context (a table lookup in shared
// memory), its state (a shuffle), the decision.
// The decoded bits go out as masks per bit-plane, and a second kernel turns
// a block's masks into coefficients (t1_coefficients_kernel).
#include <cuda_runtime.h>

#include <cstring>

#include "jp2g_internal.h"
#include "kernels.h"
#include "t1_logic.h"

namespace jp2g {

namespace {

constexpr uint32_t kCtxZC0 = 0, kCtxAGG = 17, kCtxUNI = 18;

struct DecTables {
  uint8_t zc[4 * 512];
  uint8_t sc[256];
  uint8_t spb[256];
  uint32_t mq[94];  // qe | next-MPS index << 16 | next-LPS index << 24; index = 2 state + MPS
};
__constant__ DecTables c_dec;

constexpr int kDecWarps = 4;
constexpr uint32_t kDecStates = 94;

// Context word: Qe << 15 | state << 3 | MPS. The table holds per state (state,
// MPS pair) the words after an MPS and an LPS renormalisation.
struct DecShared {
  uint2 next[kDecStates];
  uint8_t zc[4][512];  // zero-coding context by neighbourhood (neighbour_index)
  uint8_t sc[256];     // sign context | prediction bit << 7 (cross_index)
};
__device__ __forceinline__ uint32_t dec_word(uint32_t state) {
  return (c_dec.mq[state] & 0xffffu) << 15 | state << 3 | (state & 1u);
}
// The tables in the layouts used here, from those of c_dec (src/tier1/
// consts.rs: zero coding bit 0 NW, 1 N, 2 NE, 3 W, 5 E, 6 SW, 7 S, 8 SE; sign
// coding bit 3 W, 0 W negative, 1 N, 4 N negative, 5 E, 2 E negative, 7 S, 6 S
// negative).
__device__ __forceinline__ void load_dec_shared(DecShared& sh) {
  for (uint32_t i = threadIdx.x; i < kDecStates; i += blockDim.x)
    sh.next[i] = make_uint2(dec_word((c_dec.mq[i] >> 16) & 0xffu), dec_word(c_dec.mq[i] >> 24));
  for (uint32_t i = threadIdx.x; i < 4 * 512; i += blockDim.x) {
    const uint32_t f = i & 511u;
    const uint32_t g = (f & 1u) | (f >> 3 & 1u) << 1 | (f >> 6 & 1u) << 2 | (f >> 1 & 1u) << 3 | (f >> 7 & 1u) << 5 |
                       (f >> 2 & 1u) << 6 | (f >> 5 & 1u) << 7 | (f >> 8 & 1u) << 8;
    sh.zc[i >> 9][f] = c_dec.zc[(i & ~511u) | g];
  }
  for (uint32_t i = threadIdx.x; i < 256; i += blockDim.x) {
    const uint32_t s = i & 15u, g = i >> 4;  // W, N, E, S
    const uint32_t lu = (s & 1u) << 3 | (s & g & 1u) | (s >> 1 & 1u) << 1 | ((s & g) >> 1 & 1u) << 4 |
                        (s >> 2 & 1u) << 5 | ((s & g) >> 2 & 1u) << 2 | (s >> 3 & 1u) << 7 | ((s & g) >> 3 & 1u) << 6;
    sh.sc[i] = (uint8_t)(c_dec.sc[lu] | c_dec.spb[lu] << 7);
  }
}

// Six rows of a column of a stripe (bits 1..4 the stripe's, 0 and 5 the rows
// above and below it) beside its two neighbours': bits 0..5 the column to
// the west, 11..16 the column, 22..27 the one to the east (the spacing lets
// two shifts gather three bits of each).
__device__ __forceinline__ uint32_t window(uint32_t west, uint32_t own, uint32_t east) {
  return west | own << 11 | east << 22;
}
__device__ __forceinline__ uint32_t own_rows(uint32_t win) { return (win >> 12) & 0xfu; }
// Neighbourhood of row r: bits NW, W, SW, N, (itself), S, NE, E, SE.
__device__ __forceinline__ uint32_t neighbour_index(uint32_t win, int r) {
  const uint32_t t = (win >> r) & 0x01c03807u;
  return (t | t >> 8 | t >> 16) & 0x1ffu;
}
// The four direct neighbours of row r: bits W, N, E, S.
__device__ __forceinline__ uint32_t cross_index(uint32_t win, int r) {
  const uint32_t t = (win >> r) & 0x00802802u;
  return ((t | t >> 9 | t >> 20) >> 1) & 0xfu;
}
// Rows of the column with a significant neighbour.
__device__ __forceinline__ uint32_t rows_near(uint32_t win) {
  const uint32_t s = (win | win >> 22) & 0x3fu, m = (win >> 11) & 0x3fu;
  return ((s | s << 1 | s >> 1 | m << 1 | m >> 1) >> 1) & 0xfu;
}

constexpr uint32_t kAll = 0xffffffffu;

// One of a lane's two columns.
struct Column {
  unsigned long long sig, sgn, vis, ref;
  unsigned long long ones;  // the bit-plane's decoded 1 bits
};
// Rows 4 k - 1 .. 4 k + 4 of a mask.
__device__ __forceinline__ uint32_t six_rows(unsigned long long v, int k) {
  return (uint32_t)(k > 0 ? v >> (4 * k - 1) : v << 1) & 0x3fu;
}
__device__ __forceinline__ uint32_t four_rows(unsigned long long v, int k) { return (uint32_t)(v >> (4 * k)) & 0xfu; }

template <bool kMany>
struct BlockDecoder {
  const DecShared& sh;
  const uint8_t* zc;
  uint8_t* list;  // of the warp, in shared memory
  uint32_t lane;
  int w, h;
  // the MQ decoder (ISO/IEC 15444-1 C.3; src/mq/mod.rs:38-160), the same in
  // all lanes: A << 15 and C >> 1 (its lowest bit is always 0), so that a
  // difference's sign bit compares; cur and nxt are the segment's bytes bp and
  // bp + 1, 0xFF beyond its end
  const uint8_t* b;
  uint32_t n, bp, cur, nxt, a, c;
  int ct;               // below 0: C is still to be shifted, from shift_from by `shift`
  uint32_t shift_from;
  int shift;
  uint32_t word, mps_next, lps_next;  // this lane's context, and its successors
  Column col[2];

  __device__ __forceinline__ uint32_t at(uint32_t i) const { return i < n ? b[i] : 0xffu; }
  __device__ __forceinline__ void bytein() {
    if (cur == 0xffu && nxt > 0x8fu) {
      c += 0x7f80u;
      ct = 8;
    } else {
      c = (c + (cur == 0xffu ? nxt << 8 : nxt << 7)) & 0x7fffffffu;
      ct = cur == 0xffu ? 7 : 8;
      ++bp;
      cur = nxt;
      nxt = at(bp + 1);
    }
  }
  __device__ __forceinline__ void start(const uint8_t* data, uint32_t len) {
    // initial context states (src/mq/mod.rs:195-200)
    const uint32_t st = lane == kCtxUNI ? 92u : lane == kCtxAGG ? 6u : lane == kCtxZC0 ? 8u : 0u;
    word = dec_word(st);
    mps_next = sh.next[st].x;
    lps_next = sh.next[st].y;
    b = data;
    n = len;
    bp = 0;
    cur = at(0);
    nxt = at(1);
    c = cur << 15;
    bytein();
    c <<= 7;
    ct -= 7;
    a = 0x40000000u;
  }
  // After A -= Qe the coder takes Qe when C lies below it, else A (and takes
  // Qe off C); the decision is the LPS when that differs from A < Qe, and the
  // context moves on when the result is renormalised. The comparisons are
  // masks (a predicate takes longer to reach its users than a sign bit), and
  // the bytes that a shift has run out of are read at the next symbol, while
  // its context is on its way.
  // In batches, where other warps fill a chain's waits, the shortest code
  // decides instead (kMany): a decision without renormalisation ends early, and
  // the rest is predicated. A lone chain takes 13 % longer that way; 12
  // 1275x1650 files of 2x2 checks at quality 20, whose samples nearly all become
  // significant in one pass, 4.56 ms (6.6 in the other form, 4.78 with two
  // blocks to a warp, a lane each).
  __device__ __forceinline__ bool decode(uint32_t cx) {
    const uint32_t e = __shfl_sync(kAll, word, (int)cx);
    if (kMany) {
      const uint32_t qe = e & 0x7fff8000u, d = a - qe, t = c - qe;
      if ((int)((d << 1) & ~t) < 0) {  // an MPS, A still 0x8000 or more
        a = d;
        c = t;
        return (e & 1u) != 0;
      }
      const bool low = (int)t < 0, lps = low != (d < qe);
      const uint32_t v = low ? qe : d;
      if (!low) c = t;
      if (lane == cx) {
        word = lps ? lps_next : mps_next;
        const uint2 n = *reinterpret_cast<const uint2*>(reinterpret_cast<const uint8_t*>(sh.next) + (word & 0x3f8u));
        mps_next = n.x;
        lps_next = n.y;
      }
      int k = __clz((int)v) - 1;
      a = v << k;
      while (k > ct) {
        c = (c << ct) & 0x7fffffffu;
        k -= ct;
        bytein();
      }
      c = (c << k) & 0x7fffffffu;
      ct -= k;
      return ((e & 1u) != 0) != lps;
    }
    if (ct < 0) {
      c = shift_from;
      ct += shift;
      int k = shift;
      while (k > ct) {
        c = (c << ct) & 0x7fffffffu;
        k -= ct;
        bytein();
      }
      c = (c << k) & 0x7fffffffu;
      ct -= k;
    }
    const uint32_t qe = e & 0x7fff8000u;
    const uint32_t d = a - qe, t = c - qe;
    const uint32_t low = (uint32_t)((int)t >> 31), lps = low ^ (uint32_t)((int)(d - qe) >> 31);
    const uint32_t move = (low | ((d >> 30) - 1u)) & (lane == cx ? kAll : 0u);
    word = (((lps_next & lps) | (mps_next & ~lps)) & move) | (word & ~move);
    if (move) {
      const uint2 n = *reinterpret_cast<const uint2*>(reinterpret_cast<const uint8_t*>(sh.next) + (word & 0x3f8u));
      mps_next = n.x;
      lps_next = n.y;
    }
    const uint32_t v = (qe & low) | (d & ~low);
    shift_from = (c & low) | (t & ~low);
    shift = __clz((int)v) - 1;
    a = v << shift;
    c = (shift_from << shift) & 0x7fffffffu;
    ct -= shift;
    return ((e ^ lps) & 1u) != 0;
  }

  // The windows in a mask of the half's columns (half 0: columns 0..31).
  __device__ __forceinline__ uint32_t windows(int half, unsigned long long m0, unsigned long long m1, int k) const {
    const uint32_t r0 = six_rows(m0, k), r1 = six_rows(m1, k), own = half ? r1 : r0;
    uint32_t west = __shfl_up_sync(kAll, own, 1), east = __shfl_down_sync(kAll, own, 1);
    const uint32_t edge = __shfl_sync(kAll, half ? r0 : r1, half ? 31 : 0);
    if (lane == 0) west = half ? edge : 0u;
    if (lane == 31) east = half ? 0u : edge;
    return window(west, own, east);
  }

  // A column's plan: a byte for each of its rows to be coded, in order:
  // context, row << 5, and kLast in the last one. Lanes make the plans of 32
  // columns at once, so that most symbols (those of columns with no new
  // significant sample beside or above them) find their context made.
  static constexpr uint32_t kLast = 0x80u;
  static constexpr uint32_t kRunPlan = kLast | kCtxAGG;
  template <class F>
  __device__ __forceinline__ uint32_t plan_of(uint32_t rows, F context) const {
    uint32_t plan = 0;
    #pragma unroll
    for (int r = 3; r >= 0; --r)
      if ((rows >> r) & 1u) plan = plan << 8 | (plan ? 0u : kLast) | (uint32_t)r << 5 | context(r);
    return plan;
  }
  __device__ __forceinline__ uint32_t zero_plan(uint32_t win, uint32_t rows) const {
    return plan_of(rows, [&](int r) { return (uint32_t)zc[neighbour_index(win, r)]; });
  }

  // Significance propagation (clean false) or cleanup of 32 columns of a
  // stripe, `cand` the columns still to come. (One copy of the code for both
  // passes and both halves: with one each, warps in different passes ran out
  // of instruction cache, 18.6 against 13.7 ms for a 12-page batch.)
  __device__ __forceinline__ void zero_coding(int half, int k, uint32_t valid, bool clean) {
    const bool inside = (int)lane + 32 * half < w;
    uint32_t win = windows(half, col[0].sig, col[1].sig, k);
    const uint32_t vis = four_rows(half ? col[1].vis : col[0].vis, k);
    uint32_t todo = inside ? (clean ? ~vis : rows_near(win)) & ~own_rows(win) & valid : 0u;
    uint32_t cand = __ballot_sync(kAll, todo != 0);
    if (cand == 0) return;
    // in cleanup, four rows with nothing significant around are a run
    // (src/tier1/flags.rs:219-235)
    uint32_t plan_me = clean && todo == 0xfu && win == 0 ? kRunPlan : zero_plan(win, todo);
    uint32_t gwin = windows(half, col[0].sgn, col[1].sgn, k);
    uint32_t fresh_me = 0, neg_me = 0;
    do {
      const int x = __ffs((int)cand) - 1;
      cand &= cand - 1;
      uint32_t plan = __shfl_sync(kAll, plan_me, x);
      bool bit;
      #pragma unroll 1
      for (;;) {
        bit = decode(plan & 0x1fu);
        if (bit || (plan & kLast)) break;
        plan >>= 8;
      }
      if (!bit) continue;
      // the rest of the column, its window changing with each new sample
      uint32_t r = (plan >> 5) & 3u, fresh = 0, neg = 0;
      const uint32_t pair = __shfl_sync(kAll, win | todo << 28, x), gn = __shfl_sync(kAll, gwin, x);
      uint32_t wn = pair & 0x0fffffffu, td = pair >> 28;
      if (plan == kRunPlan) {
        r = 0;
        #pragma unroll 1
        for (int i = 0; i < 2; ++i) r = r << 1 | (decode(kCtxUNI) ? 1u : 0u);
      }
      #pragma unroll 1
      while (bit) {
        const uint32_t sc = sh.sc[cross_index(wn, (int)r) | cross_index(gn | neg << 12, (int)r) << 4];
        neg |= ((decode(sc & 0x7fu) ? 1u : 0u) ^ (sc >> 7)) << r;
        fresh |= 1u << r;
        wn |= 0x1000u << r;
        uint32_t rest = (clean ? td : rows_near(wn) & ~own_rows(wn) & valid) & (0xeu << r);
        td = (td & ~(0xeu << r)) | rest;  // coded, or to be coded
        bit = false;
        #pragma unroll 1
        while (rest && !bit) {
          r = (uint32_t)__ffs((int)rest) - 1;
          rest &= rest - 1;
          bit = decode(zc[neighbour_index(wn, (int)r)]);
        }
      }
      if ((int)lane == x) {
        fresh_me = fresh;
        neg_me = neg;
        todo = td;
      } else if ((int)lane == x + 1) {  // the column to the east sees them
        win |= fresh << 1;
        gwin |= neg << 1;
        if (!clean) todo = inside ? rows_near(win) & ~own_rows(win) & valid : 0u;
        plan_me = zero_plan(win, todo);
      }
      if (!clean) cand = __ballot_sync(kAll, todo != 0) & (0xfffffffeu << x);
    } while (cand);
    const unsigned long long f = (unsigned long long)fresh_me << (4 * k), g = (unsigned long long)neg_me << (4 * k),
                             v = clean ? 0ull : (unsigned long long)todo << (4 * k);
    #pragma unroll
    for (int i = 0; i < 2; ++i) {
      const bool it = i == half;
      col[i].sig |= it ? f : 0ull;
      col[i].ones |= it ? f : 0ull;
      col[i].sgn |= it ? g : 0ull;
      col[i].vis |= it ? v : 0ull;
    }
  }

  // Refinement changes no context but its own, so the contexts of a stripe's
  // 32 columns are listed in shared memory first, and what is left per symbol
  // is its decision.
  __device__ __forceinline__ void refinement(int half, int k) {
    const uint32_t win = windows(half, col[0].sig, col[1].sig, k);
    const uint32_t todo = own_rows(win) & ~four_rows(half ? col[1].vis : col[0].vis, k);
    const uint32_t in[4] = {__ballot_sync(kAll, (todo & 1u) != 0), __ballot_sync(kAll, (todo & 2u) != 0),
                            __ballot_sync(kAll, (todo & 4u) != 0), __ballot_sync(kAll, (todo & 8u) != 0)};
    const int total = __popc(in[0]) + __popc(in[1]) + __popc(in[2]) + __popc(in[3]);
    if (total == 0) return;
    // contexts 14 + (a significant neighbour), 16 once refined
    const uint32_t near = rows_near(win), ref = four_rows(half ? col[1].ref : col[0].ref, k), before = (1u << lane) - 1u;
    const int first = __popc(in[0] & before) + __popc(in[1] & before) + __popc(in[2] & before) + __popc(in[3] & before);
    int at_row = first;
    #pragma unroll
    for (int r = 0; r < 4; ++r)
      if ((todo >> r) & 1u) list[at_row++] = (uint8_t)((ref >> r) & 1u ? 16u : 14u + ((near >> r) & 1u));
    __syncwarp();
    int i = 0;
    #pragma unroll 1
    for (; i + 4 <= total; i += 4) {
      const uint32_t four = *reinterpret_cast<const uint32_t*>(list + i);
      uint32_t got = 0;
      #pragma unroll
      for (int j = 0; j < 4; ++j) got |= decode((four >> (8 * j)) & 0xffu) ? 1u << j : 0u;
      if (lane == 0) list[i >> 2] = (uint8_t)got;  // in the place of a context that has been read
    }
    if (i < total) {
      uint32_t four = *reinterpret_cast<const uint32_t*>(list + i), got = 0;
      #pragma unroll 1
      for (int j = i; j < total; ++j, four >>= 8) got |= decode(four & 0xffu) ? 1u << (j & 3) : 0u;
      if (lane == 0) list[i >> 2] = (uint8_t)got;
    }
    __syncwarp();
    uint32_t bits = (uint32_t)(list[first >> 2] | list[(first >> 2) + 1] << 4) >> (first & 3), ones = 0;
    #pragma unroll
    for (int r = 0; r < 4; ++r)
      if ((todo >> r) & 1u) {
        ones |= (bits & 1u) << r;
        bits >>= 1;
      }
    __syncwarp();
    #pragma unroll
    for (int i = 0; i < 2; ++i) {
      col[i].ones |= i == half ? (unsigned long long)ones << (4 * k) : 0ull;
      col[i].ref |= i == half ? (unsigned long long)todo << (4 * k) : 0ull;
    }
  }

  // pass 0 significance propagation, 1 refinement, 2 cleanup
  __device__ __forceinline__ void run_pass(int pass) {
    const int halves = w > 32 ? 2 : 1, parts = halves * ((h + 3) / 4);
    #pragma unroll 1
    for (int part = 0; part < parts; ++part) {
      const int k = halves == 2 ? part >> 1 : part, half = halves == 2 ? part & 1 : 0;
      const uint32_t valid = h - 4 * k >= 4 ? 0xfu : (1u << (h - 4 * k)) - 1u;
      if (pass == 1) refinement(half, k);
      else zero_coding(half, k, valid, pass == 2);
    }
    if (pass == 2) col[0].vis = col[1].vis = 0;
  }
};

// Seven CTAs fit an SM with or without the bound; with it the compiler keeps
// everything in 72 registers (without, it spills 8 bytes on the chain): a gray
// 2550x3300 file 5.36 -> 5.08 ms, a 512x512 lossless one 4.56 -> 4.34.
template <bool kMany>
__global__ void __launch_bounds__(kDecWarps * 32, 7) t1_decode_kernel(const DecBlock* blocks, const uint32_t* order,
                                                                      uint32_t nblocks, const uint8_t* data,
                                                                      unsigned long long* masks) {
  __shared__ DecShared sh;
  __shared__ __align__(4) uint8_t lists[kDecWarps][132];
  load_dec_shared(sh);
  __syncthreads();
  const uint32_t lane = threadIdx.x & 31, slot = blockIdx.x * kDecWarps + (threadIdx.x >> 5);
  if (slot >= nblocks) return;
  const DecBlock d = blocks[order[slot]];
  if (d.npasses == 0) return;
  BlockDecoder<kMany> dec{sh, sh.zc[d.orient & 3], lists[threadIdx.x >> 5], lane, d.w, d.h};
  dec.start(data + d.data_off, d.data_len);
  unsigned long long* out = masks + d.mask_off;
  // cleanup of the top bit-plane, then significance, refinement and cleanup
  // per bit-plane until the block's passes end
  int left = d.npasses, pass = 2;
  while (left > 0) {
    dec.run_pass(pass);
    --left;
    if (pass == 2 || left == 0) {  // the bit-plane's masks
      if ((int)lane < d.w) out[lane] = dec.col[0].ones;
      if ((int)lane + 32 < d.w) out[lane + 32] = dec.col[1].ones;
      dec.col[0].ones = dec.col[1].ones = 0;
      out += d.w;
    }
    pass = pass == 2 ? 0 : pass + 1;
  }
  if ((int)lane < d.w) out[lane] = dec.col[0].sgn;
  if ((int)lane + 32 < d.w) out[lane + 32] = dec.col[1].sgn;
}

// Coefficients of every code-block from its masks, a warp per block: a lane
// takes 32 rows of a column, and a 32x32 bit transpose in registers turns its
// bit-planes into magnitudes. Signed integers (reversible codestreams) or
// midpoint-dequantised values (sign * (|q| + 0.5) * step,
// src/simd/scalar.rs:122-129).
// (Bound by the latency of its loads and stores: at five CTAs per SM 12 sRGB
// 2550x3300 files take 0.45 ms, at the three of 141 registers 0.52.)
__global__ void __launch_bounds__(128, 5) t1_coefficients_kernel(const DecBlock* blocks, uint32_t nblocks,
                                                                 const unsigned long long* masks, int32_t* planes) {
  const int lane = threadIdx.x & 31;
  const uint32_t b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (b >= nblocks) return;
  const DecBlock d = blocks[b];
  int32_t* plane = planes + d.plane_off;
  const int top = (int)d.mb - (int)d.zbp - 1, np = (int)dec_planes(d.npasses);
  const uint32_t* mw = reinterpret_cast<const uint32_t*>(masks + d.mask_off);
  #pragma unroll 1
  for (int x = lane; x < d.w; x += 32)
    #pragma unroll 1
    for (int half = 0; 32 * half < d.h; ++half) {
      uint32_t t[32];
      #pragma unroll
      for (int k = 0; k < 32; ++k) {
        const int j = top - k;  // bit-plane k is the block's plane j
        t[k] = j >= 0 && j < np ? mw[(d.w * j + x) * 2 + half] : 0u;
      }
      const uint32_t sg = np > 0 ? mw[(d.w * np + x) * 2 + half] : 0u;
      transpose32(t);
      #pragma unroll
      for (int i = 0; i < 32; ++i) {
        const int y = 32 * half + i;
        if (y >= d.h) break;
        const bool neg = (sg >> i) & 1u;
        int32_t v = neg ? -(int32_t)t[i] : (int32_t)t[i];
        if (!d.reversible) {
          float f = 0.0f;
          if (t[i] != 0) f = __fmul_rn(__fmul_rn(neg ? -1.0f : 1.0f, __fadd_rn((float)t[i], 0.5f)), d.step);
          v = __float_as_int(f);
        }
        plane[(size_t)y * d.stride + x] = v;
      }
    }
}

// Decoding order: longest segments first (counting sort on 1024 buckets of 16
// bytes), so that the longest chains start first.
constexpr uint32_t kDecBuckets = 1024;
__device__ __forceinline__ uint32_t dec_bucket(const DecBlock& d) {
  return kDecBuckets - 1 - min(d.data_len >> 4, kDecBuckets - 1);
}
__global__ void dec_hist_kernel(const DecBlock* blocks, uint32_t n, uint32_t* hist) {
  const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b < n) atomicAdd(hist + dec_bucket(blocks[b]), 1u);
}
__global__ void dec_scatter_kernel(const DecBlock* blocks, uint32_t n, uint32_t* cursor, uint32_t* order) {
  const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b < n) order[atomicAdd(cursor + dec_bucket(blocks[b]), 1u)] = b;
}

}  // namespace

bool upload_decode_tables(const uint8_t* zc, const uint8_t* sc, const uint8_t* spb, const uint32_t* mq) {
  DecTables t;
  memcpy(t.zc, zc, sizeof t.zc);
  memcpy(t.sc, sc, sizeof t.sc);
  memcpy(t.spb, spb, sizeof t.spb);
  memcpy(t.mq, mq, sizeof t.mq);
  return cudaMemcpyToSymbol(c_dec, &t, sizeof t) == cudaSuccess;
}

void launch_t1_decode(const DecBlock* blocks, uint32_t nblocks, const uint8_t* data, unsigned long long* masks,
                      int32_t* planes, uint32_t* scratch, bool many, cudaStream_t st) {
  if (nblocks == 0) return;
  uint32_t* hist = scratch;
  uint32_t* cursor = scratch + kDecBuckets;
  uint32_t* order = scratch + 2 * kDecBuckets;
  cudaMemsetAsync(hist, 0, kDecBuckets * sizeof(uint32_t), st);
  const uint32_t g = (nblocks + 255) / 256;
  dec_hist_kernel<<<g, 256, 0, st>>>(blocks, nblocks, hist);
  launch_scan_u32(hist, 1, kDecBuckets - 1, cursor, order, st);  // `order` is filled after the scan
  dec_scatter_kernel<<<g, 256, 0, st>>>(blocks, nblocks, cursor, order);
  const uint32_t ctas = (nblocks + kDecWarps - 1) / kDecWarps;
  if (many) t1_decode_kernel<true><<<ctas, kDecWarps * 32, 0, st>>>(blocks, order, nblocks, data, masks);
  else t1_decode_kernel<false><<<ctas, kDecWarps * 32, 0, st>>>(blocks, order, nblocks, data, masks);
  t1_coefficients_kernel<<<(nblocks + 3) / 4, 128, 0, st>>>(blocks, nblocks, masks, planes);
}

}  // namespace jp2g
