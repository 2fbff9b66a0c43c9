// bp_quad.cu -- backprojection of slice stacks, four slices at a time (sm_100a).
//
// The slices of a stack share angles, centre and output grid, so they share the
// sample index of every update.  The filter stores four slices interleaved (one
// 16-byte word per sample, fbp_kernels.hpp), and one index and one shared-memory
// load then serve four updates.  With truncation, arithmetic and accumulation order per
// pixel are those of bp_fast.cu -- the reference's (ctas src/common/lct.cpp:688-729,
// ct.cl:14-43) -- bit for bit.  Linear interpolation adds one interpolated sample per
// projection where bp_fast.cu sums samples and differences apart, so a slice's rounding
// there depends on whether it is in a group (the error against 64 bits is the same,
// 2.0e-5 on 900 x 1536).
//
// What bounds it.  One slice at a time (bp_fast.cu) every update costs a 4-byte shared
// load and an index: 4.1 instructions and 1.0 wavefronts per 32 updates, 1569 us per
// slice of 1800 x 2560 (tile 15; 20.3 updates per clock and SM).  Here 2.1 instructions
// and 0.59 wavefronts, 847 us (37.6): shared-memory wavefronts 69 % of their peak,
// issue 64 %, FMA and integer pipes 56 % each, none of which leaves much.
//   * 16-byte loads of interleaved slices: 4 wavefronts serve 128 updates and the index
//     arithmetic is shared, but alone they leave the wavefront bound where it was
//     (1.0 per 32 updates): 1082 us.
//   * A thread owns blocks of 4 x 2 neighbouring pixels, and pixels whose sample must be
//     one of two that their neighbours load take it by a select (sharing patterns,
//     below): 0.49 loads per pixel.
//   * Lanes arranged so that the eight of a wavefront span at most eight words: bank
//     conflicts 17 % of the wavefronts -> 1 %, 907 -> 847 us.
//   * No producer warp: nine warps of a CTA leave 96 registers a thread, eight 128, and
//     the accumulators alone take 64.  The warps take turns at issuing the copies
//     (one warp that issues them all is always the last: 1023 -> 941 us).
//   * 32 projections a stage in 2 stages rather than 16 in 4: 949 -> 896 us.
// The loop over projections is not unrolled: a pass is 130 instructions for each of 12
// patterns and layouts, and twice that no longer stays in the instruction cache
// (2398 us with 4 warps a CTA).  Half the pixels per thread, 24 warps an SM: 998 us.
// QSmall keeps that register limit (three CTAs), but with 32 projections a stage its
// windows leave room for two.
// Linear interpolation (an extension, FP64-derived projection bases) uses the same
// layouts and patterns with two loads per sample: 397 instead of 980 us per slice of
// 900 x 1536, bound by registers (its samples, differences and fractions).
#include <cuda_runtime.h>

#include <cstdint>
#include <cstdio>

#include "bp_common.cuh"
#include "bp_quad.hpp"
#include "bp_quad_rule.hpp"
#include "bp_stage.cuh"

namespace ctas {
namespace {

constexpr int kChunk = 32;  // projections per pipeline stage
constexpr int kStages = 2;
typedef unsigned long long u64;

thread_local char t_detail[160];

// CTA tile: WX x WY warps of 16 columns x 16 UB rows.
template <int WX_, int WY_, int UB_, int BOX_, int MINB_> struct QTile {
  static constexpr int WX = WX_, WY = WY_, UB = UB_, BOX = BOX_, MINB = MINB_;
  static constexpr int TX = 16 * WX, TY = 16 * UB * WY, WARPS = WX * WY, THREADS = 32 * WARPS;
  // window span (TY-1)|sin| + (TX-1)|cos|, start 2 below the lowest index, rounding
  static_assert((BOX - 6) * (BOX - 6) >= (TY - 1) * (TY - 1) + (TX - 1) * (TX - 1),
                "window too short for the tile");
  static_assert(BOX <= kQuadSlack, "windows stay within the buffer's slack");
};
using QLarge = QTile<4, 2, 2, 96, 2>;  // 64 x 64, 16 pixels per thread
using QSmall = QTile<4, 2, 1, 80, 3>;  // 32 x 64, 8 pixels per thread

struct __align__(16) Param {
  float sx, cy, base;  // sin, cos, c + ((1 - sin) - cos) * hp, times 2^-22; linear
                       // interpolation: sin, cos, t0
  float m;             // 2 + (window word address - window start) * 2^-22; linear
                       // interpolation: the bits of the window's address bias
};

template <class TL> struct Layout {
  float4 win[kStages][kChunk][TL::BOX];
  Param par[kStages][kChunk];
  uint4 ctl[kStages];  // x: pixel layout; y, z, w: bit planes of the sharing patterns
  uint32_t neg[kStages];  // wide layout: projections whose indices may be negative
  float xch[TL::WARPS][256];
  u64 full[kStages], empty[kStages];
  int active[TL::WARPS];
  int rank[TL::WARPS];  // number of a warp among those with pixels in the disc
  int nactive;
};

__device__ __forceinline__ void add64(u64 &a, u64 w) {
  asm("add.rn.f32x2 %0, %0, %1;" : "+l"(a) : "l"(w));
}

// a += (ka == kb) ? w : v, for two pairs.  Selects and two adds; four predicated
// packed adds instead ran 24 % slower (more instructions).
__device__ __forceinline__ void add64_eq(u64 &a0, u64 &a1, uint32_t ka, uint32_t kb, const u64 *w,
                                         const u64 *v) {
  const bool same = ka == kb;
  add64(a0, same ? w[0] : v[0]);
  add64(a1, same ? w[1] : v[1]);
}

__device__ __forceinline__ void lds_quad(uint32_t addr, u64 *w) {
  asm("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(w[0]), "=l"(w[1]) : "r"(addr));
}

// x << 4 as a funnel shift with a low word below 2^28 (integer ALU)
__device__ __forceinline__ uint32_t shl4_alu(uint32_t x, uint32_t lo) {
  uint32_t r;
  asm("shf.l.wrap.b32 %0, %1, %2, 4;" : "=r"(r) : "r"(lo), "r"(x));
  return r;
}

__device__ __forceinline__ float2 both(float v) { return make_float2(v, v); }

// Pixel layouts.  A warp owns 16 x 32 pixels, two blocks u of 16 x 16 one below the
// other; a thread owns 4 x 2 pixels of each, pixel 4 r + k at
//   slow = 4 hi + k (15 less that if mirrored), fast = 2 lo + r,
// slow and fast being column and row (bit 0 clear) or row and column (bit 0 set).
// slow is the axis along which t moves less, and mirroring makes t move the same
// way along k and r, so within a thread t = t0 +- (k u + r s), 0 <= u <= s: the
// closer two pixels are, the likelier they read the same sample.  Eight
// consecutive lanes share a wavefront of 16-byte loads, without bank conflicts where
// their samples span at most eight words.  They are 2 slow x 4 fast neighbours, or with
// kSkew, for u > s / 3, eight of equal or neighbouring 1.25 hi + lo, whose t hardly
// differs: no conflicts, where the 2 x 4 neighbours cost 7 to 19 % more wavefronts (and
// kSkew, near the axes, 17 to 40 %).
constexpr int kRow = 1, kMirror = 2, kSkew = 4;  // bits of a layout
constexpr int kLayouts = 8;
template <int UB> using Acc = u64[UB][8][2];  // [u][pixel][slices 0-1, 2-3]

// 8 hi + lo of each lane, and the lane of each 8 hi + lo
__constant__ unsigned char kSkewPlace[32] = {0, 1, 8, 2, 9, 16, 3, 10, 17, 24, 4, 11, 18, 25, 5, 12, 19, 26, 6, 13, 20, 27, 7, 14, 21, 28, 15, 22, 29, 23, 30, 31};
__constant__ unsigned char kSkewLane[32] = {0, 1, 3, 6, 10, 14, 18, 22, 2, 4, 7, 11, 15, 19, 23, 26, 5, 8, 12, 16, 20, 24, 27, 29, 9, 13, 17, 21, 25, 28, 30, 31};
__device__ __forceinline__ int place_of_lane(int layout, int lane) {
  if (layout & kSkew) return kSkewPlace[lane];
  return ((lane >> 2) & 3) * 8 + ((lane >> 4) << 2 | (lane & 3));
}
__device__ __forceinline__ int lane_of_place(int layout, int hi, int lo) {
  if (layout & kSkew) return kSkewLane[8 * hi + lo];
  return (lo >> 2) << 4 | hi << 2 | (lo & 3);
}

// Sharing patterns: which pixels load their sample, and for each of the others two
// loaded pixels A, B with t between theirs and theirs less than 1 apart, so that its
// index is A's or B's.  The order of t along k or r alone survives rounding (sums
// of rounded terms are monotone); any other order, and every distance, needs the
// margin m, above the rounding error of two values of t.  Loads per eight pixels:
// 3 where 3u <= s (A), 4 up to 2u = s (B) and up to 3u - s = 1 (C), 5 beyond (D); on
// average over a half turn 0.49 of the pixels.
constexpr int kPatterns = 6;
struct Share {
  signed char a, b;  // -1: loads its own sample
};
__host__ __device__ constexpr Share share(int pattern, int px) {
  constexpr Share L{-1, -1};
  constexpr Share t[kPatterns][8] = {
      {L, L, L, L, L, L, L, L},                                // every pixel loads
      {L, {0, 4}, {4, 5}, L, L, L, {3, 7}, L},                 // D
      {L, {0, 4}, {4, 3}, L, L, {4, 3}, {3, 7}, L},            // C
      {L, {0, 4}, {0, 4}, {4, 6}, L, {4, 6}, L, L},            // B
      {L, {0, 4}, {0, 4}, {0, 4}, L, {4, 7}, {4, 7}, L},       // A
      {L, {0, 3}, {0, 3}, L, L, {4, 7}, {4, 7}, L}};           // runs along k alone
  return t[pattern][px];
}
__device__ __forceinline__ int pattern_of(float u, float s, float m) {
  const float one = 1.0f - m;
  if (s <= one && u + m <= s) {
    if (3.f * u <= one && 3.f * u + m <= s) return 4;
    if (2.f * u <= one && 2.f * u + m <= s && s + m <= 3.f * u) return 3;
    if (s + m <= 2.f * u) return 3.f * u - s <= one ? 2 : 1;
  }
  return 3.f * u <= one ? 5 : 0;
}

// One projection.  cA: coordinates along slow (pairs k, k + 1; for rows of both
// blocks), cB: along fast (pairs r).
template <int UB, bool ROW, int PAT, bool NEG, bool kCheck>
__device__ __forceinline__ void project(const Param &p, const float2 (&cA)[2 * UB],
                                        const float2 (&cB)[UB], Acc<UB> &acc, uint32_t lo_bits,
                                        uint32_t win, uint32_t win_bytes, int *err) {
  const float2 m2 = both(p.m);
  float2 slow[ROW ? 2 * UB : 2], fast[ROW ? 1 : UB];
  if constexpr (ROW) {
#pragma unroll
    for (int q = 0; q < 2 * UB; q++) slow[q] = add2_rn(both(p.base), mul2z_rn(both(p.sx), cA[q]));
    fast[0] = mul2z_rn(both(p.cy), cB[0]);
  } else {
#pragma unroll
    for (int q = 0; q < 2; q++) slow[q] = mul2z_rn(both(p.cy), cA[q]);
#pragma unroll
    for (int q = 0; q < UB; q++) fast[q] = add2_rn(both(p.base), mul2z_rn(both(p.sx), cB[q]));
  }
#pragma unroll
  for (int u = 0; u < UB; u++) {
    uint32_t k[8];
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const float2 fr = fast[ROW ? 0 : u];
      const float2 t = add2_rn(both(q < 2 ? fr.x : fr.y), slow[(ROW ? 2 * u : 0) + (q & 1)]);
      float2 v = add2_rm(t, m2);
      if constexpr (NEG) {  // truncation: ceiling below zero
        const float2 c = add2_rp(t, m2);
        v = make_float2(t.x < 0.f ? c.x : v.x, t.y < 0.f ? c.y : v.y);
      }
      k[2 * q] = __float_as_uint(v.x);
      k[2 * q + 1] = __float_as_uint(v.y);
    }
    u64 w[8][2];
#pragma unroll
    for (int i = 0; i < 8; i++) {
      if (share(PAT, i).a >= 0) continue;
      const uint32_t a = shl4_alu(k[i], lo_bits);
      if (kCheck) {
        const bool ok = a - win < win_bytes;
        if (!ok) atomicOr(err, 8);
        w[i][0] = w[i][1] = 0;
        if (ok) lds_quad(a, w[i]);
      } else {
        lds_quad(a, w[i]);
      }
      add64(acc[u][i][0], w[i][0]);
      add64(acc[u][i][1], w[i][1]);
    }
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const int ia = share(PAT, i).a, ib = share(PAT, i).b;
      if (ia < 0) continue;
      if (kCheck && k[i] != k[ia] && k[i] != k[ib]) atomicOr(err, 8);
      add64_eq(acc[u][i][0], acc[u][i][1], k[i], k[ia], w[ia], w[ib]);
    }
  }
}

// One projection with linear interpolation: u = t0 + sin j + cos i, k = floor(u),
// q[k] + (u - k) (q[k+1] - q[k]).  Pixels that share a sample share its neighbour.
template <int UB, bool ROW, int PAT, bool kCheck>
__device__ __forceinline__ void project_linear(const Param &p, const float2 (&cA)[2 * UB],
                                               const float2 (&cB)[UB], Acc<UB> &acc, uint32_t win,
                                               uint32_t win_bytes, int *err) {
  const uint32_t bias = __float_as_uint(p.m);
  float2 rows[ROW ? 2 * UB : UB];  // t0 + sin j
#pragma unroll
  for (int q = 0; q < (ROW ? 2 * UB : UB); q++)
    rows[q] = fma2_rn(both(p.sx), ROW ? cA[q] : cB[ROW ? 0 : q], both(p.base));
#pragma unroll
  for (int u = 0; u < UB; u++) {
    uint32_t k[8];
    float f[8];
#pragma unroll
    for (int q = 0; q < 4; q++) {
      float2 v;
      if constexpr (ROW) {
        v = fma2_rn(both(p.cy), both(q < 2 ? cB[0].x : cB[0].y), rows[2 * u + (q & 1)]);
      } else {
        v = fma2_rn(both(p.cy), cA[q & 1], both(q < 2 ? rows[u].x : rows[u].y));
      }
      const float2 m = add2_rm(v, both(kMagic));
      const float2 fl = add2_rn(m, both(-kMagic));
      k[2 * q] = __float_as_uint(m.x);
      k[2 * q + 1] = __float_as_uint(m.y);
      f[2 * q] = __fsub_rn(v.x, fl.x);
      f[2 * q + 1] = __fsub_rn(v.y, fl.y);
    }
    float2 w[8][2], d[8][2];  // samples and differences to the next ones
    auto add = [&](int i, int h, float2 w0, float2 w1) {
      float2 &o = *reinterpret_cast<float2 *>(&acc[u][i][h]);
      o = add2_rn(o, fma2_rn(both(f[i]), w1, w0));
    };
#pragma unroll
    for (int i = 0; i < 8; i++) {
      if (share(PAT, i).a >= 0) continue;
      const uint32_t a = (k[i] << 4) + bias;
      u64 x[2] = {0, 0}, y[2] = {0, 0};
      if (!kCheck || a - win < win_bytes - 16) {
        lds_quad(a, x);
        lds_quad(a + 16, y);
      } else {
        atomicOr(err, 8);
      }
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const float2 y2 = *reinterpret_cast<float2 *>(&y[h]);
        w[i][h] = *reinterpret_cast<float2 *>(&x[h]);
        d[i][h] = add2_rn(y2, make_float2(-w[i][h].x, -w[i][h].y));
        add(i, h, w[i][h], d[i][h]);
      }
    }
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const int ia = share(PAT, i).a, ib = share(PAT, i).b;
      if (ia < 0) continue;
      if (kCheck && k[i] != k[ia] && k[i] != k[ib]) atomicOr(err, 8);
      const bool same = k[i] == k[ia];
#pragma unroll
      for (int h = 0; h < 2; h++) add(i, h, same ? w[ia][h] : w[ib][h], same ? d[ia][h] : d[ib][h]);
    }
  }
}

// Row-major position of a thread's pixel in its 16 x 16 block; layout -1: the stores',
// which put eight consecutive columns on eight lanes.
__device__ __forceinline__ int place(int layout, int lane, int px) {
  if (layout < 0) return 16 * (4 * (lane >> 3) + (px & 3)) + 8 * (px >> 2) + (lane & 7);
  const int at = place_of_lane(layout, lane), k = px & 3;
  const int run = 4 * (at >> 3) + k, slow = (layout & kMirror) ? 15 - run : run;
  const int fast = 2 * (at & 7) + (px >> 2);
  return (layout & kRow) ? 16 * slow + fast : 16 * fast + slow;
}

// Moves the accumulators from one layout to another through the warp's buffer, which
// holds them as (pixel, lane) of the old one: the writes have no bank conflicts.
template <int UB>
__device__ __forceinline__ void exchange(Acc<UB> &acc, float *buf, int lane, int from, int to) {
  int src[8];
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const int at = place(to, lane, i), row = at >> 4, col = at & 15;
    const int slow = (from & kRow) ? row : col, fast = (from & kRow) ? col : row;
    const int run = (from & kMirror) ? 15 - slow : slow;
    src[i] = 32 * (4 * (fast & 1) + (run & 3)) + lane_of_place(from, run >> 2, fast >> 1);
  }
#pragma unroll
  for (int u = 0; u < UB; u++)
#pragma unroll
    for (int h = 0; h < 2; h++) {
      float2 v[8];
#pragma unroll
      for (int i = 0; i < 8; i++) v[i] = *reinterpret_cast<float2 *>(&acc[u][i][h]);
#pragma unroll
      for (int i = 0; i < 8; i++) buf[32 * i + lane] = v[i].x;
      __syncwarp();
#pragma unroll
      for (int i = 0; i < 8; i++) v[i].x = buf[src[i]];
      __syncwarp();
#pragma unroll
      for (int i = 0; i < 8; i++) buf[32 * i + lane] = v[i].y;
      __syncwarp();
#pragma unroll
      for (int i = 0; i < 8; i++) v[i].y = buf[src[i]];
      __syncwarp();
#pragma unroll
      for (int i = 0; i < 8; i++) acc[u][i][h] = *reinterpret_cast<u64 *>(&v[i]);
    }
}

template <class TL, bool kLinear, bool kWide, bool kCheck>
__global__ void __launch_bounds__(TL::THREADS, TL::MINB) bp_quad_kernel(BpLaunch a) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  Layout<TL> &sm = *reinterpret_cast<Layout<TL> *>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127));
  const int W = a.W, N = a.N, hp = W / 2, R = a.out_rows, C = a.out_cols;
  const float c = a.center, oj = a.geo_oj, oi = a.geo_oi, pg = a.geo_p;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int i0 = blockIdx.x * TL::TX, j0 = blockIdx.y * TL::TY;
  const int iw = i0 + 16 * (warp % TL::WX), jw = j0 + 16 * TL::UB * (warp / TL::WX);
  const int s0 = 4 * blockIdx.z, ns = min(4, a.S - s0);
  float *out = a.out + (int64_t)s0 * a.out_slice_stride;
  const uint32_t limit = a.wait_limit ? a.wait_limit : kWaitLimit;

  bool mine = false;
#pragma unroll
  for (int e = 0; e < 8 * TL::UB; e++) {
    const int at = place(-1, lane, e & 7), j = jw + 16 * (e >> 3) + (at >> 4), i = iw + (at & 15);
    mine |= (j < R && i < C) && ref_mask_f(geo(oj, pg, j), geo(oi, pg, i), W, c);
  }
  const bool act = __any_sync(0xffffffffu, mine);
  if (lane == 0) sm.active[warp] = act ? 1 : 0;
  __syncthreads();
  if (threadIdx.x == 0) {
    int n = 0;
    for (int w = 0; w < TL::WARPS; w++) {
      sm.rank[w] = n;
      n += sm.active[w];
    }
    sm.nactive = n;
    if (n) {
      for (int s = 0; s < kStages; s++) {
        mbar_init(&sm.full[s], 1);
        mbar_init(&sm.empty[s], (uint32_t)n);
      }
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
  }
  __syncthreads();
  if (!act) {
    for (int s = 0; s < ns; s++)
#pragma unroll
      for (int e = 0; e < 8 * TL::UB; e++) {
        const int at = place(-1, lane, e & 7), j = jw + 16 * (e >> 3) + (at >> 4), i = iw + (at & 15);
        if (j < R && i < C) out[s * a.out_slice_stride + (int64_t)j * C + i] = 0.f;
      }
    return;
  }

  const int nchunks = (N + kChunk - 1) / kChunk;
  // The warps take turns at issuing copies: chunk ch is copied by the warp of rank
  // ch mod (warps with pixels).  One warp that issued them all was always the last,
  // and the others waited for its copies.
  int turn = sm.rank[warp];  // next chunk this warp copies
  const int turns = sm.nactive;
  // waits (bounded) for this warp's copies still in flight
  auto drain = [&] {
    if (lane != 0) return;
    for (int d = turn - turns; d >= 0 && d > turn - turns - kStages; d -= turns)
      mbar_wait(&sm.full[d % kStages], (uint32_t)((d / kStages) & 1), limit);
  };
  // Parameters and copies of chunk `turn`; false on a timeout.
  auto produce = [&]() -> bool {
    const int ch = turn, st = ch % kStages;
    if (ch >= kStages && !mbar_wait(&sm.empty[st], (uint32_t)(((ch / kStages) - 1) & 1), limit))
      return false;
    const int n = ch * kChunk + lane, cnt = min(kChunk, N - ch * kChunk);
    const bool live = lane < cnt;
    float2 sc = make_float2(0.f, 0.f);
    int x0 = 0;
    float tmin = 0.f;
    if (live) {
      const float ja = geo(oj, pg, j0), jb = geo(oj, pg, j0 + TL::TY - 1);
      const float ia = geo(oi, pg, i0), ib = geo(oi, pg, i0 + TL::TX - 1);
      Param p;
      if constexpr (kLinear) {
        // u = t - 0.5, t0 formed in FP64
        const double2 g = a.lin[n];
        const double hc = (double)hp + (double)c;
        p.sx = sc.x = (float)g.x;
        p.cy = sc.y = (float)g.y;
        p.base = (float)(hc * (1.0 - g.x) - g.y * (double)hp - 0.5);
        x0 = window_start_linear(p.sx, p.cy, p.base, ja, jb, ia, ib, 1);
        p.m = __uint_as_float(smem_u32(&sm.win[st][lane][0]) - 16u * (kMagicBits + (uint32_t)x0));
      } else {
        sc = a.tab[n];
        const float base = ref_base(sc.x, sc.y, hp, c, a.rule);
        x0 = window_start_trunc(sc.x, sc.y, base, ja, jb, ia, ib, c, 1, &tmin);
        // off = window word address - x0, |off| < 2^22: M is exact
        const int off = (int)(smem_u32(&sm.win[st][lane][0]) >> 4) - x0;
        p.sx = __fmul_rn(sc.x, kTwoM22);
        p.cy = __fmul_rn(sc.y, kTwoM22);
        p.base = __fmul_rn(base, kTwoM22);
        p.m = __fadd_rn(2.0f, __fmul_rn((float)off, kTwoM22));
      }
      sm.par[st][lane] = p;
    }
    // the layout that most of the chunk's projections want
    const bool row = fabsf(sc.x) < fabsf(sc.y);
    const float margin = (float)(W + 256) * 1.9073486328125e-06f;  // (W + 256) 2^-19
    const float su = fminf(fabsf(sc.x), fabsf(sc.y)) * pg, ss = fmaxf(fabsf(sc.x), fabsf(sc.y)) * pg;
    const int want = (row ? kRow : 0) | ((sc.x < 0.f) != (sc.y < 0.f) ? kMirror : 0) |
                     (3.f * su > ss ? kSkew : 0);
    int copy_layout = 0, most = -1;
#pragma unroll
    for (int l = 0; l < kLayouts; l++) {
      const int votes = __popc(__ballot_sync(0xffffffffu, live && want == l));
      if (votes > most) {
        most = votes;
        copy_layout = l;
      }
    }
    // another layout than a projection's own leaves it the runs along k alone
    const float run = ((copy_layout & kRow) ? fabsf(sc.x) : fabsf(sc.y)) * pg;
    const int pat = !live ? 0
                    : ((want ^ copy_layout) & (kRow | kMirror)) == 0
                        ? pattern_of(su, ss, margin)
                        : (3.f * run <= 1.0f - margin ? 5 : 0);
    const uint32_t b0 = __ballot_sync(0xffffffffu, pat & 1), b1 = __ballot_sync(0xffffffffu, pat & 2),
                   b2 = __ballot_sync(0xffffffffu, pat & 4);
    // projections for which some pixel of the tile may have t < 0
    const uint32_t neg = kWide ? __ballot_sync(0xffffffffu, live && tmin < 1.0f) : 0u;
    if (lane == 0) {
      sm.ctl[st] = make_uint4((uint32_t)copy_layout, b0, b1, b2);
      sm.neg[st] = neg;
    }
    __syncwarp();
    if (lane == 0) mbar_arrive_expect_tx(&sm.full[st], (uint32_t)(cnt * TL::BOX * sizeof(float4)));
    __syncwarp();
    if (live && !(a.test_stall && ch == 0)) {
      // within the rows and their slack; otherwise the copy is left out, and the
      // stage times out instead of faulting
      const int64_t Wp = a.Wp, rows = (int64_t)N * ((a.S + 3) / 4);
      const int64_t at = ((int64_t)blockIdx.z * N + n) * Wp + (a.off ? a.off : kRowOff) + x0;
      if (at >= -kQuadSlack && at + TL::BOX <= rows * Wp + kQuadSlack)
        bulk_load(&sm.win[st][lane][0], reinterpret_cast<const float4 *>(a.q) + at,
                  TL::BOX * sizeof(float4), &sm.full[st]);
      else
        atomicOr(a.err, 16);
    }
    turn += turns;
    return true;
  };
  while (turn < min(kStages - 1, nchunks)) produce();  // no waits yet

  Acc<TL::UB> acc;
#pragma unroll
  for (int e = 0; e < 16 * TL::UB; e++) (&acc[0][0][0])[e] = 0;
  float2 cA[2 * TL::UB], cB[TL::UB];
  auto jc = [&](int j) { return kLinear ? geo(oj, pg, j) : __fsub_rn(geo(oj, pg, j), c); };
  auto coords = [&](int layout) {
    const int hi = place_of_lane(layout, lane) >> 3, lo = place_of_lane(layout, lane) & 7;
    auto slow = [&](int k) { return (layout & kMirror) ? 15 - (4 * hi + k) : 4 * hi + k; };
    if (layout & kRow) {
#pragma unroll
      for (int q = 0; q < 2 * TL::UB; q++) {
        const int j = jw + 16 * (q >> 1), k = 2 * (q & 1);
        cA[q] = make_float2(jc(j + slow(k)), jc(j + slow(k + 1)));
      }
#pragma unroll
      for (int q = 0; q < TL::UB; q++)
        cB[q] = make_float2(geo(oi, pg, iw + 2 * lo), geo(oi, pg, iw + 2 * lo + 1));
    } else {
#pragma unroll
      for (int q = 0; q < 2 * TL::UB; q++)
        cA[q] = make_float2(geo(oi, pg, iw + slow(2 * (q & 1))), geo(oi, pg, iw + slow(2 * (q & 1) + 1)));
#pragma unroll
      for (int q = 0; q < TL::UB; q++)
        cB[q] = make_float2(jc(jw + 16 * q + 2 * lo), jc(jw + 16 * q + 2 * lo + 1));
    }
  };
  int layout = 0;
  coords(layout);
  const uint32_t lo_bits = threadIdx.x;  // any value below 2^28 the compiler cannot fold away

  for (int ch = 0; ch < nchunks; ch++) {
    const int st = ch % kStages;
    if (!mbar_wait(&sm.full[st], (uint32_t)((ch / kStages) & 1), limit)) {
      if (lane == 0) atomicOr(a.err, 4);
      drain();
      return;
    }
    const int cnt = min(kChunk, N - ch * kChunk);
    const uint4 ctl = sm.ctl[st];
    if ((int)ctl.x != layout) {
      exchange<TL::UB>(acc, sm.xch[warp], lane, layout, (int)ctl.x);
      layout = (int)ctl.x;
      coords(layout);
    }
    // stretches of projections of one pattern; the first half of the chunk apart, so
    // that the next copies are issued half a chunk after this warp's release of
    // their stage, when the other warps have released it too
    const uint32_t neg = kWide ? sm.neg[st] : 0u;
    const uint32_t change = ((ctl.y ^ (ctl.y >> 1)) | (ctl.z ^ (ctl.z >> 1)) | (ctl.w ^ (ctl.w >> 1)) |
                             (neg ^ (neg >> 1)) | (1u << (cnt / 2) >> 1)) &
                            ((1u << (cnt - 1)) - 1u);
    for (int k = 0; k < cnt;) {
      if (k == cnt / 2 && turn == ch + kStages - 1 && turn < nchunks && !produce()) {
        if (lane == 0) atomicOr(a.err, 4);
        drain();
        return;
      }
      const uint32_t rest = change >> k;
      const int end = rest ? k + __ffs(rest) : cnt;
      auto go = [&](auto row, auto pat, auto ng) {
        constexpr bool ROW = decltype(row)::value;
        [[maybe_unused]] constexpr bool NEG = decltype(ng)::value;
        constexpr int PAT = decltype(pat)::value;
        const Param *pp = &sm.par[st][k];
#pragma unroll 1
        for (int n = k; n < end; n++) {
          const Param p = *pp++;
          const uint32_t win = kCheck ? smem_u32(&sm.win[st][n][0]) : 0u;
          if constexpr (kLinear)
            project_linear<TL::UB, ROW, PAT, kCheck>(p, cA, cB, acc, win, TL::BOX * 16, a.err);
          else
            project<TL::UB, ROW, PAT, NEG, kCheck>(p, cA, cB, acc, lo_bits, win, TL::BOX * 16, a.err);
        }
      };
      auto pick = [&](auto row, auto ng) {
        switch (((ctl.y >> k) & 1u) | (((ctl.z >> k) & 1u) << 1) | (((ctl.w >> k) & 1u) << 2)) {
        case 1: return go(row, std::integral_constant<int, 1>{}, ng);
        case 2: return go(row, std::integral_constant<int, 2>{}, ng);
        case 3: return go(row, std::integral_constant<int, 3>{}, ng);
        case 4: return go(row, std::integral_constant<int, 4>{}, ng);
        case 5: return go(row, std::integral_constant<int, 5>{}, ng);
        default: return go(row, std::integral_constant<int, 0>{}, ng);
        }
      };
      if (kWide && ((neg >> k) & 1u)) {
        if (layout & kRow) pick(std::true_type{}, std::true_type{});
        else pick(std::false_type{}, std::true_type{});
      } else {
        if (layout & kRow) pick(std::true_type{}, std::false_type{});
        else pick(std::false_type{}, std::false_type{});
      }
      k = end;
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&sm.empty[st]);
  }

  exchange<TL::UB>(acc, sm.xch[warp], lane, layout, -1);
#pragma unroll
  for (int u = 0; u < TL::UB; u++)
#pragma unroll
    for (int e = 0; e < 8; e++) {
      const int at = place(-1, lane, e), j = jw + 16 * u + (at >> 4), i = iw + (at & 15);
      if (j >= R || i >= C) continue;
      const bool in = ref_mask_f(geo(oj, pg, j), geo(oi, pg, i), W, c);
      float *o = out + (int64_t)j * C + i;
#pragma unroll
      for (int s = 0; s < 4; s++) {
        const u64 v = acc[u][e][s >> 1];
        const float f = __uint_as_float((uint32_t)((s & 1) ? (v >> 32) : v));
        if (s < ns) o[s * a.out_slice_stride] = in ? ref_finish(f, a.rec_cof, N) : 0.f;
      }
    }
}

template <class TL, bool kLinear, bool kWide, bool kCheck>
cudaError_t launch(const BpLaunch &a, cudaStream_t st) {
  auto kern = bp_quad_kernel<TL, kLinear, kWide, kCheck>;
  const size_t smem = sizeof(Layout<TL>) + 128;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
  if (e == cudaSuccess) {
    const dim3 grid((a.out_cols + TL::TX - 1) / TL::TX, (a.out_rows + TL::TY - 1) / TL::TY,
                    (a.S + 3) / 4);
    kern<<<grid, TL::THREADS, smem, st>>>(a);
    e = cudaGetLastError();
  }
  if (e != cudaSuccess)
    std::snprintf(t_detail, sizeof(t_detail), "four-slice launch of tile %dx%d (%d threads, %zu B): %s",
                  TL::TY, TL::TX, TL::THREADS, smem, cudaGetErrorString(e));
  return e;
}

template <class TL> cudaError_t launch_form(const BpLaunch &a, cudaStream_t st, bool check) {
  if (a.interp == 1)
    return check ? launch<TL, true, false, true>(a, st) : launch<TL, true, false, false>(a, st);
  if (a.wide)
    return check ? launch<TL, false, true, true>(a, st) : launch<TL, false, true, false>(a, st);
  return check ? launch<TL, false, false, true>(a, st) : launch<TL, false, false, false>(a, st);
}

}  // namespace

const char *bp_quad_error_detail() { return t_detail; }

cudaError_t launch_bp_quad(const BpLaunch &a, cudaStream_t st, bool check) {
  t_detail[0] = 0;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (a.interp == 1 && a.wide) return cudaErrorInvalidValue;
  const int64_t tiles = (int64_t)((a.out_rows + QLarge::TY - 1) / QLarge::TY) *
                        ((a.out_cols + QLarge::TX - 1) / QLarge::TX) * ((a.S + 3) / 4);
  return quad_small_tile(tiles, sms) ? launch_form<QSmall>(a, st, check)
                                     : launch_form<QLarge>(a, st, check);
}

}  // namespace ctas
