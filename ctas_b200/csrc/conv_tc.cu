// conv_tc.cu -- 3x3 convolution of the learned stage as an implicit GEMM on the
// fifth-generation tensor cores (tcgen05.mma, accumulators in tensor memory).
//
// GEMM view of one output tile: D[128 pixels][NT channels] += A_t[128][K] * B_t[NT][K]^T
// over the nine taps t = (ky, kx) and the input channels in chunks of CK, where
// A_t row m is input pixel (y0 + m/16 + ky - 1, x0 + m%16 + kx - 1) of an 8 x 16
// pixel block and B_t row n is w[n][t][.].  Both operands are K-major (channels
// contiguous, NHWC activations and [cout][9][cin] weights) and reach shared memory
// by TMA with the hardware swizzle the matrix descriptors expect (128 B rows for
// CK = 64, 64 B for 32, 32 B for 16):
//
//   A: one 10 x 16 pixel box x CK channels per (kx, chunk) -- rows y0-1 .. y0+8,
//      zero-filled outside the image by the TMA unit -- serves the three ky taps:
//      tap ky's 128 x CK operand is the same box shifted by 16 ky rows, which
//      keeps every operand start on a swizzle-atom boundary;
//   B: the weights viewed as a 2-D array [cout][9 cin]; three NT x CK boxes per
//      (kx, chunk), one per ky tap, placed one after another -- loaded once and kept
//      where all of them fit beside the input boxes and a CTA has several tiles, else
//      with each input box.
//
// Persistent warp-specialised CTA (192 threads): warp 0 issues the TMA loads
// into a ring of stages, warp 1 issues the MMAs (K = 16 each) and releases each
// stage with tcgen05.commit, warps 2-5 drain the accumulator (tcgen05.ld, bias, ReLU
// or ReLU mask, BF16) through shared memory into TMA stores while the next tile
// accumulates in another tensor-memory buffer.  Every wait is bounded; on expiry the
// kernel records an error, drains its copies and MMAs, frees its tensor memory and
// returns.
//
// What bounds it: the operands' shared-memory reads (128 x 16 and NT x 16 elements per
// MMA: 48 clocks for N = 64, whose math takes 32) and, for 16 and 32 input channels,
// the epilogue's latency per tile.  Measured steps, with the same outputs bit for bit:
//   * the issuing warp stays converged and one elected lane issues each MMA, so that
//     descriptors and counters live in uniform registers: a single thread took about 100
//     clocks per MMA to form them;
//   * outputs through TMA stores (drain32), and a wait's limit loaded only when its first
//     try fails;
//   * in the row form below the ring's segments as plain scalars (403 -> 312 us on 96 -> 32
//     at 2048 x 2048).  Together the row form went from 270 to 169 us on 64 -> 64 at
//     2 x 1024 x 1024, and at 2048 x 2048 from 528 to 312 on 96 -> 32, 207 to 129 on
//     32 -> 32 and 180 to 115 on 16 -> 32;
//   * resident weights, and all of tensor memory for the only CTA of an SM.
// The tiled form with resident weights runs 64 -> 64 in 171 us and 96 -> 32 in 342, no
// faster than the row form, and it adds a pixel's products in another order, which
// changes the BF16 rounding of every layer after it: a layer keeps its form.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <type_traits>

#include "../../include/ctas_learned.h"
#include "../../include/ctas_fbp.h"
#include "tma_encode.hpp"
#include "unet_kernels.hpp"

namespace ctas {
namespace {

using bf16 = __nv_bfloat16;

constexpr int kThreads = 192;
constexpr uint32_t kWaitLimit = 1u << 22;
constexpr int kMaxCout = 512;

constexpr int kOutBytes = 32 * 32 * 2;  // 2 rows of 16 pixels x 32 channels

struct TcArgs {
  const bf16 *mask;
  int m_cs, m_co;
  const float *bias;
  int cout;
  int relu;
  int H, W;
  int tiles_x, tiles_y, tiles_n;
  int64_t total;
  int cin;
  int kchunks;  // cin / CK
  int stages;   // resident weights: stages of input boxes
  int *err;     // bit 0: a bounded wait ran out
};

// ST stages of (input box, weight boxes); ST = 0: the weights of all taps and chunks
// stay in shared memory and a stage, of which there are TcArgs::stages, holds an input
// box alone
template <int CK, int NT, int ST> struct TcCfg {
  static constexpr bool kResident = ST == 0;
  static constexpr int kABytes = 160 * CK * 2;     // 10 x 16 pixels x CK channels
  static constexpr int kBBytes = 3 * NT * CK * 2;  // three ky taps x NT x CK
  static constexpr int kStage = kResident ? kABytes : kABytes + kBBytes;
  static constexpr int kRowB = CK * 2;             // bytes per operand row
  static constexpr int kSBO = 8 * kRowB;           // bytes between 8-row groups
  // descriptor layout type: 128 B / 64 B / 32 B swizzle
  static constexpr uint64_t kLayout = CK == 64 ? 2 : CK == 32 ? 4 : 6;
  // accumulator buffers in tensor memory: as many as fit 256 columns (two CTAs
  // per SM), so the MMAs run ahead of the epilogue on small tiles
  static constexpr int kAcc = 256 / NT >= 8 ? 8 : 256 / NT >= 4 ? 4 : 2;
  static constexpr uint32_t kCols = 256;
  // barriers and two words, bias of all output channels, alignment slack
  static constexpr int kMaxStages = kResident ? 8 : ST;
  static constexpr int kBias = 512, kFixed = kBias + 4 * kMaxCout + 1024;
  static_assert((2 * kMaxStages + 2 * kAcc + 2) * 8 + 8 <= kBias, "barriers run into the bias");
  // output staging of each epilogue warp: buffers of 32 pixels x 32 channels, two where
  // a tile fills several (96 -> 32 runs 418 instead of 342 us with a second one, which
  // costs it a stage of input)
  static constexpr int kOutBufs = NT == 32 ? 1 : 2;
  static constexpr int kOut = 4 * kOutBufs * kOutBytes;
  static constexpr int smem(int stages, int kchunks) {
    return stages * kStage + (kResident ? 3 * kchunks * kBBytes : 0) + kOut + kFixed;
  }
  static_assert(kABytes % 1024 == 0 && kBBytes % 1024 == 0, "stage alignment");
  static_assert(NT % 32 == 0 && NT >= 32 && NT <= 128, "UMMA N, epilogue pairs");
};

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count)
               : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Test aid (ctas_nn_test_timeout): while g_test_stall is set, each kernel's
// producer leaves its first stage of copies out, so the waits on it run out;
// g_wait_limit bounds every wait (short while the test aid is armed).
__device__ int g_test_stall = 0;
__device__ uint32_t g_wait_limit = kWaitLimit;

// bounded wait; false when the limit ran out.  The limit is read after a first try:
// its load would stand before every wait that is already over.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity) {
  if (mbar_try_wait(bar, parity)) return true;
  const uint32_t limit = __ldg(&g_wait_limit);
  for (uint32_t it = 0; it < limit; ++it)
    if (mbar_try_wait(bar, parity)) return true;
  return false;
}

__device__ __forceinline__ void tma_load_4d(void *dst, const CUtensorMap *map, int c0, int c1,
                                            int c2, int c3, uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(c3),
      "r"(smem_u32(bar))
      : "memory");
}

__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *map, int c0, int c1,
                                            uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3}], [%4];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(smem_u32(bar))
      : "memory");
}

// shared -> global copy of a box, one bulk group
__device__ __forceinline__ void tma_store_4d(const CUtensorMap *map, const void *src, int c0, int c1,
                                             int c2, int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%1, %2, %3, %4}], [%5];" ::"l"(
          reinterpret_cast<uint64_t>(map)),
      "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(smem_u32(src))
      : "memory");
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}

__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// D[tmem] (+)= A[desc] * B[desc]^T, kind::f16 (BF16 operands, FP32 accumulate), by a
// whole converged warp, whose elected lane issues: descriptors and loop counters stay
// warp-uniform, in uniform registers.
__device__ __forceinline__ void tc_mma_w(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc,
                                         uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p, e;\n elect.sync _|e, 0xffffffff;\n setp.ne.b32 p, %4, 0;\n"
      " @e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
      "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tc_commit_w(uint64_t *bar) {
  asm volatile(
      "{\n .reg .pred e;\n elect.sync _|e, 0xffffffff;\n"
      " @e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}\n" ::"r"(
          smem_u32(bar))
      : "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, "
      "%11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}

__device__ __forceinline__ void tmem_wait_ld() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// shared-memory matrix descriptor of a K-major swizzled operand
template <class C> __device__ __forceinline__ uint64_t sdesc(uint32_t addr) {
  return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)1 << 16) |
         ((uint64_t)((C::kSBO >> 4) & 0x3FFF) << 32) | ((uint64_t)1 << 46) |
         (C::kLayout << 61);
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t *>(&v);
}

// Epilogue step of one warp: 32 columns of its 32 accumulator rows (one pixel a lane) ->
// bias, ReLU or mask -> BF16 in the staging buffer `so`, 64-byte rows in the 64-byte
// swizzle of the store's tensor map.  Waits until at most PENDING earlier stores
// still read their buffers.  A thread holds one pixel's channels, so its own global
// stores would put every lane of a 16-byte store on another line, 32 wavefronts each.
template <int PENDING>
__device__ __forceinline__ void drain32(uint32_t taddr, const float *bias, const bf16 *mask, int relu,
                                        uint8_t *so, int lane) {
  // two 16-column loads in flight per wait
  uint32_t r[2][16];
  tmem_ld16(taddr, r[0]);
  tmem_ld16(taddr + 16u, r[1]);
  uint4 mk[4];
  if (mask) {
#pragma unroll
    for (int h = 0; h < 4; h++) mk[h] = *reinterpret_cast<const uint4 *>(mask + 8 * h);
  }
  if (lane == 0) asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(PENDING) : "memory");
  __syncwarp();
  tmem_wait_ld();
#pragma unroll
  for (int h = 0; h < 4; h++) {  // 8 channels, one 16-byte word
    float v[8];
#pragma unroll
    for (int j = 0; j < 8; j++) {
      v[j] = __uint_as_float(r[h >> 1][8 * (h & 1) + j]) + bias[8 * h + j];
      if (relu) v[j] = fmaxf(v[j], 0.f);
    }
    if (mask) {
      const bf16 *mm = reinterpret_cast<const bf16 *>(&mk[h]);
#pragma unroll
      for (int j = 0; j < 8; j++)
        if (!(__bfloat162float(mm[j]) > 0.f)) v[j] = 0.f;
    }
    uint4 o;
    o.x = pack_bf16(v[0], v[1]);
    o.y = pack_bf16(v[2], v[3]);
    o.z = pack_bf16(v[4], v[5]);
    o.w = pack_bf16(v[6], v[7]);
    *reinterpret_cast<uint4 *>(so + lane * 64 + ((h ^ ((lane >> 1) & 3)) << 4)) = o;
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  __syncwarp();
}

struct Tile {
  int b, ty, tx, nt;
};

__device__ __forceinline__ Tile decode(const TcArgs &a, int64_t t) {
  Tile r;
  r.nt = (int)(t % a.tiles_n);
  t /= a.tiles_n;
  r.tx = (int)(t % a.tiles_x);
  t /= a.tiles_x;
  r.ty = (int)(t % a.tiles_y);
  r.b = (int)(t / a.tiles_y);
  return r;
}


template <int CK, int NT, int ST>
__global__ void __launch_bounds__(kThreads, 1)
    conv_tc_kernel(const __grid_constant__ CUtensorMap amap,
                   const __grid_constant__ CUtensorMap bmap,
                   const __grid_constant__ CUtensorMap ymap, TcArgs a) {
  using C = TcCfg<CK, NT, ST>;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t pad = (1024u - (smem_u32(smem_raw) & 1023u)) & 1023u;
  uint8_t *base = smem_raw + pad;
  const int nst = C::kResident ? a.stages : ST;
  uint8_t *wts = base + nst * C::kStage;  // resident weights: [chunk][kx][ky] blocks
  uint8_t *outs = wts + (C::kResident ? 3 * a.kchunks * C::kBBytes : 0);
  uint8_t *bars = outs + C::kOut;
  uint64_t *full = reinterpret_cast<uint64_t *>(bars);
  uint64_t *empty = full + nst;
  uint64_t *acc_full = empty + nst;  // [kAcc]
  uint64_t *acc_empty = acc_full + C::kAcc;
  uint64_t *drain = acc_empty + C::kAcc;
  uint64_t *wfull = drain + 1;  // resident weights have landed
  uint32_t *s_tmem = reinterpret_cast<uint32_t *>(wfull + 1);
  volatile int *s_abort = reinterpret_cast<volatile int *>(s_tmem + 1);
  float *s_bias = reinterpret_cast<float *>(bars + C::kBias);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < nst; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(wfull, 1);
    for (int i = 0; i < C::kAcc; i++) {
      mbar_init(&acc_full[i], 1);
      mbar_init(&acc_empty[i], 128);
    }
    mbar_init(drain, 1);
    *s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(s_tmem)),
                 "r"(C::kCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  for (int c = threadIdx.x; c < a.cout; c += kThreads) s_bias[c] = a.bias ? a.bias[c] : 0.f;
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *s_tmem;
  const int ksteps = 3 * a.kchunks;

  if (warp == 0) {
    if (lane == 0) {
      // ------------------------------------------------ TMA producer
      asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&amap))
                   : "memory");
      asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&bmap))
                   : "memory");
      int stage = 0;
      uint32_t ph = 0;
      uint32_t issued = 0, last_par = 0;  // per-stage bits: used / parity of last issue
      if constexpr (C::kResident) {
        mbar_expect_tx(wfull, (uint32_t)(3 * a.kchunks * C::kBBytes));
        for (int i = 0; i < 9 * a.kchunks; i++) {  // block (chunk, kx, ky)
          const int ky = i % 3, kx = i / 3 % 3, kc = i / 9;
          tma_load_2d(wts + i * NT * C::kRowB, &bmap, (ky * 3 + kx) * a.cin + kc * CK, 0, wfull);
        }
      }
      for (int64_t t = blockIdx.x; t < a.total && !*s_abort; t += gridDim.x) {
        const Tile tl = decode(a, t);
        for (int ks = 0; ks < ksteps; ks++) {
          const int kc = ks / 3, kx = ks % 3;
          if (!mbar_wait(&empty[stage], ph ^ 1)) {
            atomicOr(a.err, 1);
            *s_abort = 1;
            break;
          }
          uint8_t *sa = base + stage * C::kStage;
          mbar_expect_tx(&full[stage], (uint32_t)C::kStage);
          if (!(t == blockIdx.x && ks == 0 && __ldg(&g_test_stall))) {
            tma_load_4d(sa, &amap, kc * CK, tl.tx * 16 + kx - 1, tl.ty * 8 - 1, tl.b, &full[stage]);
            if constexpr (!C::kResident) {
#pragma unroll
              for (int ky = 0; ky < 3; ky++)
                tma_load_2d(sa + C::kABytes + ky * NT * C::kRowB, &bmap,
                            (ky * 3 + kx) * a.cin + kc * CK, tl.nt * NT, &full[stage]);
            }
          }
          issued |= 1u << stage;
          last_par = (last_par & ~(1u << stage)) | (ph << stage);
          if (++stage == nst) {
            stage = 0;
            ph ^= 1;
          }
        }
      }
      // every issued copy has landed before the CTA may exit
      for (int s = 0; s < nst; s++)
        if ((issued >> s) & 1u)
          if (!mbar_wait(&full[s], (last_par >> s) & 1u)) atomicOr(a.err, 1);
      if (C::kResident && !mbar_wait(wfull, 0)) atomicOr(a.err, 1);
    }
  } else if (warp == 1) {
    {
      // ------------------------------------------------ MMA issuer (whole warp)
      constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(NT >> 3) << 17) |
                                 ((uint32_t)(128 >> 4) << 24);
      int stage = 0;
      uint32_t ph = 0;
      int acc = 0;
      uint32_t acc_ph = 0;
      if (C::kResident && !__all_sync(0xffffffffu, mbar_wait(wfull, 0)) && lane == 0) {
        atomicOr(a.err, 1);
        *s_abort = 1;
      }
      __syncwarp();
      for (int64_t t = blockIdx.x; t < a.total && !__shfl_sync(0xffffffffu, *s_abort, 0); t += gridDim.x) {
        if (!__all_sync(0xffffffffu, mbar_wait(&acc_empty[acc], acc_ph ^ 1))) {
          if (lane == 0) {
            atomicOr(a.err, 1);
            *s_abort = 1;
          }
          break;
        }
        tc_fence_after();
        const uint32_t d = tmem + (uint32_t)(acc * NT);
        bool ok = true;
        for (int ks = 0; ks < ksteps; ks++) {
          if (!__all_sync(0xffffffffu, mbar_wait(&full[stage], ph))) {
            if (lane == 0) {
              atomicOr(a.err, 1);
              *s_abort = 1;
            }
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t sa = smem_u32(base + stage * C::kStage);
          const uint64_t da = sdesc<C>(sa),
                         db = sdesc<C>(C::kResident ? smem_u32(wts) + ks * C::kBBytes : sa + C::kABytes);
#pragma unroll
          for (int ky = 0; ky < 3; ky++)
#pragma unroll
            for (int kk = 0; kk < CK / 16; kk++)
              tc_mma_w(d, da + (uint64_t)((ky * 16 * C::kRowB + kk * 32) >> 4),
                     db + (uint64_t)((ky * NT * C::kRowB + kk * 32) >> 4), idesc,
                     (ks | ky | kk) != 0 ? 1u : 0u);
          tc_commit_w(&empty[stage]);  // the stage is free once these MMAs have read it
          if (++stage == nst) {
            stage = 0;
            ph ^= 1;
          }
        }
        if (!ok) break;
        tc_commit_w(&acc_full[acc]);
        if (++acc == C::kAcc) {
          acc = 0;
          acc_ph ^= 1;
        }
      }
      // all MMAs of this thread complete before tensor memory is released
      tc_commit_w(drain);
      if (!mbar_wait(drain, 0)) atomicOr(a.err, 1);
    }
  } else {
    // ---------------------------------------------------- epilogue (warps 2-5)
    const int q = warp & 3;  // tensor-memory lane quarter this warp may access
    const int m = q * 32 + lane;
    int acc = 0, turn = 0;
    uint32_t acc_ph = 0;
    for (int64_t t = blockIdx.x; t < a.total; t += gridDim.x) {
      // warp-uniform decisions: the tensor-memory loads below are warp-collective
      if (__shfl_sync(0xffffffffu, *s_abort, 0)) break;
      if (!__all_sync(0xffffffffu, mbar_wait(&acc_full[acc], acc_ph))) {
        if (lane == 0) {
          atomicOr(a.err, 1);
          *s_abort = 1;
        }
        break;
      }
      tc_fence_after();
      const Tile tl = decode(a, t);
      const int yy = tl.ty * 8 + (m >> 4), xx = tl.tx * 16 + (m & 15);
      const int64_t pix = ((int64_t)tl.b * a.H + yy) * a.W + xx;
      const bf16 *mp = a.mask ? a.mask + pix * a.m_cs + a.m_co + tl.nt * NT : nullptr;
      const float *bp = s_bias + tl.nt * NT;
      const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(acc * NT);
#pragma unroll 1
      for (int c0 = 0; c0 < NT; c0 += 32, turn ^= 1) {
        uint8_t *so = outs + (C::kOutBufs == 2 ? 2 * q + turn : q) * kOutBytes;
        drain32<C::kOutBufs - 1>(taddr + (uint32_t)c0, bp + c0, mp ? mp + c0 : nullptr, a.relu, so, lane);
        if (lane == 0) tma_store_4d(&ymap, so, tl.nt * NT + c0, tl.tx * 16, tl.ty * 8 + 2 * q, tl.b);
      }
      tc_fence_before();
      mbar_arrive(&acc_empty[acc]);
      if (++acc == C::kAcc) {
        acc = 0;
        acc_ph ^= 1;
      }
    }
    // the staging buffers are read before the CTA may exit
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }

  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(C::kCols)
                 : "memory");
}

// ------------------------------------------------------------ host side
using EncodeTiledFn = ctas::EncodeTiledFn;
EncodeTiledFn encode_fn() { return ctas::tensor_map_encoder(); }

CUtensorMapSwizzle swizzle_for(int ck) {
  return ck == 64 ? CU_TENSOR_MAP_SWIZZLE_128B
                  : ck == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B;
}

// activations: (cin, W, H, B) of the channel slice; box {CK, 16, 10, 1}
bool make_act_map(const ConvArgs &a, int ck, CUtensorMap *map) {
  EncodeTiledFn enc = encode_fn();
  if (!enc) return false;
  std::memset(map, 0, sizeof(*map));
  const cuuint64_t dims[4] = {(cuuint64_t)a.cin, (cuuint64_t)a.W, (cuuint64_t)a.H,
                              (cuuint64_t)a.B};
  const cuuint64_t cs = (cuuint64_t)a.x_cs * 2;
  const cuuint64_t strides[3] = {cs, cs * (cuuint64_t)a.W, cs * (cuuint64_t)a.W * a.H};
  const cuuint32_t box[4] = {(cuuint32_t)ck, 16u, 10u, 1u};
  const cuuint32_t estr[4] = {1u, 1u, 1u, 1u};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<bf16 *>(a.x + a.x_co), dims,
             strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle_for(ck),
             CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) ==
         CUDA_SUCCESS;
}

// outputs: (cout, W, H, B) of the channel slice; box {32, bw, bh, 1}, bw * bh = 32
bool make_out_map(const ConvArgs &a, int bw, int bh, CUtensorMap *map) {
  EncodeTiledFn enc = encode_fn();
  if (!enc) return false;
  std::memset(map, 0, sizeof(*map));
  const cuuint64_t dims[4] = {(cuuint64_t)a.cout, (cuuint64_t)a.W, (cuuint64_t)a.H,
                              (cuuint64_t)a.B};
  const cuuint64_t cs = (cuuint64_t)a.y_cs * 2;
  const cuuint64_t strides[3] = {cs, cs * (cuuint64_t)a.W, cs * (cuuint64_t)a.W * a.H};
  const cuuint32_t box[4] = {32u, (cuuint32_t)bw, (cuuint32_t)bh, 1u};
  const cuuint32_t estr[4] = {1u, 1u, 1u, 1u};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, a.y + a.y_co, dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B,
             CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) ==
         CUDA_SUCCESS;
}

// weights [cout][9][cin] as a 2-D array (9 cin, cout); box {CK, NT}
bool make_wt_map(const ConvArgs &a, int ck, int nt, CUtensorMap *map) {
  EncodeTiledFn enc = encode_fn();
  if (!enc) return false;
  std::memset(map, 0, sizeof(*map));
  const cuuint64_t dims[2] = {9 * (cuuint64_t)a.cin, (cuuint64_t)a.cout};
  const cuuint64_t strides[1] = {9 * (cuuint64_t)a.cin * 2};
  const cuuint32_t box[2] = {(cuuint32_t)ck, (cuuint32_t)nt};
  const cuuint32_t estr[2] = {1u, 1u};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<bf16 *>(a.w), dims, strides,
             box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle_for(ck),
             CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) ==
         CUDA_SUCCESS;
}

// device error word of the tensor-core convolutions (mapped host memory, so
// the host reads it without a device synchronisation)
int *g_err_host = nullptr;
int *g_err_dev = nullptr;
std::mutex g_err_mutex;

cudaError_t err_word(int **dev) {
  std::lock_guard<std::mutex> l(g_err_mutex);
  if (!g_err_host) {
    void *p = nullptr;
    cudaError_t e = cudaHostAlloc(&p, sizeof(int), cudaHostAllocMapped | cudaHostAllocPortable);
    if (e != cudaSuccess) return e;
    *static_cast<int *>(p) = 0;
    void *d = nullptr;
    e = cudaHostGetDevicePointer(&d, p, 0);
    if (e != cudaSuccess) {
      cudaFreeHost(p);
      return e;
    }
    g_err_host = static_cast<int *>(p);
    g_err_dev = static_cast<int *>(d);
  }
  *dev = g_err_dev;
  return cudaSuccess;
}

// resident CTAs per SM for `smem` bytes of dynamic shared memory, the
// kernel's registers and `per_sm` (tensor-memory) limit
template <class K> int occupancy(K kernel, int smem, int per_sm) {
  cudaFuncAttributes fa{};
  int regs = 128;
  if (cudaFuncGetAttributes(&fa, kernel) == cudaSuccess && fa.numRegs > 0) regs = fa.numRegs;
  const int by_regs = 65536 / (((regs + 7) / 8) * 8 * kThreads);
  const int by_smem = 233472 / (smem + 1024);
  return std::max(1, std::min(per_sm, std::min(by_regs, by_smem)));
}

int sm_count() {
  static int n = 0;
  if (!n) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (n <= 0) n = 148;
  }
  return n;
}

template <int CK, int NT, int ST>
cudaError_t launch_cfg(const ConvArgs &a, cudaStream_t st) {
  using C = TcCfg<CK, NT, ST>;
  CUtensorMap amap, bmap, ymap;
  if (!make_act_map(a, CK, &amap) || !make_wt_map(a, CK, NT, &bmap) || !make_out_map(a, 16, 2, &ymap))
    return cudaErrorInvalidValue;
  TcArgs t{};
  t.mask = a.mask;
  t.m_cs = a.m_cs;
  t.m_co = a.m_co;
  t.bias = a.bias;
  t.cout = a.cout;
  t.relu = a.relu;
  t.H = a.H;
  t.W = a.W;
  t.tiles_x = a.W / 16;
  t.tiles_y = a.H / 8;
  t.tiles_n = a.cout / NT;
  t.total = (int64_t)a.B * t.tiles_y * t.tiles_x * t.tiles_n;
  t.cin = a.cin;
  t.kchunks = a.cin / CK;
  cudaError_t e = err_word(&t.err);
  if (e != cudaSuccess) return e;
  // no more CTAs per SM than tensor memory holds (512 columns): pad the
  // shared-memory request so that one more would not fit
  const int per_sm = 512 / (int)C::kCols;
  t.stages = ST;
  if (C::kResident) {
    // two CTAs per SM where three stages fit beside the weights, else one
    const int half = (233472 / 2 - 1024 - C::smem(0, t.kchunks)) / C::kStage;
    const int all = (232448 - C::smem(0, t.kchunks)) / C::kStage;
    t.stages = std::min(C::kMaxStages, half >= 3 ? half : all);
    if (t.stages < 3) return cudaErrorInvalidValue;
  }
  const int smem = std::max(C::smem(t.stages, t.kchunks), 232448 / (per_sm + 1) + 1024);
  e = cudaFuncSetAttribute(conv_tc_kernel<CK, NT, ST>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           smem);
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(conv_tc_kernel<CK, NT, ST>,
                           cudaFuncAttributePreferredSharedMemoryCarveout,
                           (int)cudaSharedmemCarveoutMaxShared);
  if (e != cudaSuccess) return e;
  const int occ = occupancy(conv_tc_kernel<CK, NT, ST>, smem, per_sm);
  const int64_t grid = std::min<int64_t>(t.total, (int64_t)sm_count() * occ);
  conv_tc_kernel<CK, NT, ST><<<(unsigned)grid, kThreads, smem, st>>>(amap, bmap, ymap, t);
  return cudaGetLastError();
}

// Whether the weights of all nine taps fit beside three input boxes (64 -> 128, 128 -> 64
// and the layers below on rows that the row form does not take): the CTAs then read
// them once instead of per tile.  64 -> 128 at 2 x 512 x 512 91 -> 70 us.  From more than
// two tiles per SM on: a CTA with one tile waits for all weights before its first MMA
// (32 -> 32 at 64 x 64 5.6 us resident and 5.3 with the input boxes, at 2 x 128 x 144 6.2
// and 5.9, at 2 x 256 x 208 8.8 and 9.3).
template <int CK, int NT> bool resident_pays(const ConvArgs &a) {
  return a.cout == NT && TcCfg<CK, NT, 0>::smem(3, a.cin / CK) <= 232448 &&
         (int64_t)a.B * (a.H / 8) * (a.W / 16) > 2 * sm_count();
}

template <int CK, int NT> cudaError_t launch_ck_nt(const ConvArgs &a, cudaStream_t st) {
  if (resident_pays<CK, NT>(a)) return launch_cfg<CK, NT, 0>(a, st);
  constexpr int kStage = 160 * CK * 2 + 3 * NT * CK * 2;
  constexpr int kSt = (96 * 1024) / kStage < 2 ? 2 : (96 * 1024) / kStage > 6 ? 6 : (96 * 1024) / kStage;
  return launch_cfg<CK, NT, kSt>(a, st);
}

template <int CK> cudaError_t launch_ck(const ConvArgs &a, int nt, cudaStream_t st) {
  switch (nt) {
    case 32: return launch_ck_nt<CK, 32>(a, st);
    case 64: return launch_ck_nt<CK, 64>(a, st);
    case 96: return launch_ck_nt<CK, 96>(a, st);
    case 128: return launch_ck_nt<CK, 128>(a, st);
    default: return cudaErrorInvalidValue;
  }
}

// ------------------------------------------------------------ row-streaming form
// For layers whose weights fit in shared memory and whose rows are multiples of
// 128 pixels (the full-resolution layers with few output channels, where the
// tiled form above reads every input pixel 3.75 times from L2 for only NT
// outputs): a CTA walks down a strip 128 pixels wide, each input row is loaded
// once into a ring of row buffers and serves the three output rows and nine
// taps that need it, and the weights stay resident.  An input row is stored as
// 64-channel chunks of 130 pixels x 128 bytes in the 128-byte-swizzled K-major
// layout (one TMA box per chunk; channels beyond cin are zero-filled by the
// TMA unit and never multiplied); the operand of tap (ky, kx) is the buffer of
// row y + ky - 1 started kx pixel rows in.  The weights are stored per (tap,
// channel chunk) as swizzled K-major blocks of cout rows (128-, 64- or 32-byte
// rows for 64-, 32- or 16-channel chunks), written by the threads with the same
// address swizzle the TMA unit applies.
constexpr int kRowPx = 130;                    // 128 output pixels + 2 halo
constexpr int kRowChunkBytes = 17 * 1024;      // 130 x 128 B, padded to the 1 KB atom
constexpr int kRowMaxSlots = 8;
constexpr int kMaxAcc = 8;
// Bias of all output channels, barriers and two words: behind the staging buffers, or with
// one buffer per epilogue warp in the padding of the first row buffer, where 64 -> 32 and
// 32 -> 64 so fit twice into an SM (115,712 bytes each): at 2 x 1024 x 1024 96 us instead
// of 139, which one CTA took, and 94 instead of 131.
constexpr int kRowMaxCout = 64;
constexpr int kRowTail = 4 * kRowMaxCout + (2 * kRowMaxSlots + 2 * kMaxAcc + 1) * 8 + 8;
constexpr int kRowPad = kRowPx * 128;          // start of that padding
static_assert(kRowPad % 16 == 0 && kRowPad + kRowTail <= kRowChunkBytes,
              "bias and barriers in the padding of a row buffer");

struct RowArgs {
  const bf16 *mask;
  int m_cs, m_co;
  const float *bias;
  const bf16 *w;  // [cout][9][cin]
  int cin, cout, relu;
  int H, W;
  int strips_x, strips_y, strip_h;
  int64_t total;  // B * strips_y * strips_x
  int nslots, slot_bytes, wbytes;
  int nacc;       // accumulator buffers in tensor memory
  uint32_t cols;
  int *err;
};

// swizzled K-major descriptor for rows of RB bytes (128, 64 or 32; 8-row groups
// 8 RB apart)
template <int RB> __device__ __forceinline__ uint64_t sdesc_swz(uint32_t addr) {
  constexpr uint64_t layout = RB == 128 ? 2 : RB == 64 ? 4 : 6;
  return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)1 << 16) | ((uint64_t)((8 * RB) >> 4) << 32) |
         ((uint64_t)1 << 46) | (layout << 61);
}

// byte offset of a swizzled operand (rows of RB bytes, region 1024-byte aligned):
// the 16-byte unit index XOR the row phase, as the hardware swizzle does
template <int RB> __host__ __device__ __forceinline__ uint32_t swz(uint32_t off) {
  constexpr uint32_t mask = RB == 128 ? 7u : RB == 64 ? 3u : 1u;
  return off ^ (((off >> 7) & mask) << 4);
}

// 128-byte-swizzled K-major descriptor (rows of 128 B, 8-row groups 1024 B apart).
// The swizzle is applied to the absolute shared-memory address (bits 4-6 XOR
// bits 7-9), as the TMA unit applies it when writing, so an operand may start
// any whole number of rows past a 1024-byte atom with the base offset left 0.
__device__ __forceinline__ uint64_t sdesc_sw128(uint32_t addr) {
  return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) |
         ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}

// BUFS: staging buffers per epilogue warp, 1 or 2
template <int CIN, int BUFS>
__global__ void __launch_bounds__(kThreads, 1)
    conv_row_kernel(const __grid_constant__ CUtensorMap amap,
                    const __grid_constant__ CUtensorMap ymap, RowArgs a) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t pad = (1024u - (smem_u32(smem_raw) & 1023u)) & 1023u;
  uint8_t *base = smem_raw + pad;
  uint8_t *slots = base;                                   // input-row ring (1 KB atoms)
  uint8_t *wsm = base + a.nslots * a.slot_bytes;           // weights
  uint8_t *outs = wsm + a.wbytes;                          // output staging
  float *s_bias = reinterpret_cast<float *>(BUFS == 1 ? base + kRowPad : outs + 4 * BUFS * kOutBytes);
  uint64_t *row_full = reinterpret_cast<uint64_t *>(s_bias + kRowMaxCout);
  uint64_t *row_empty = row_full + kRowMaxSlots;
  uint64_t *acc_full = row_empty + kRowMaxSlots;  // [kMaxAcc]
  uint64_t *acc_empty = acc_full + kMaxAcc;
  uint64_t *drain = acc_empty + kMaxAcc;
  uint32_t *s_tmem = reinterpret_cast<uint32_t *>(drain + 1);
  volatile int *s_abort = reinterpret_cast<volatile int *>(s_tmem + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ns = a.nslots, cout = a.cout;
  constexpr int cin = CIN;
  if (threadIdx.x == 0) {
    for (int s = 0; s < ns; s++) {
      mbar_init(&row_full[s], 1);
      mbar_init(&row_empty[s], 1);
    }
    for (int i = 0; i < a.nacc; i++) {
      mbar_init(&acc_full[i], 1);
      mbar_init(&acc_empty[i], 128);
    }
    mbar_init(drain, 1);
    *s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(s_tmem)),
                 "r"(a.cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  // weights -> swizzled K-major blocks [kx][chunk][3 cout rows][kCKB channels]:
  // in a block, rows p * cout + n hold tap (ky = 2 - p, kx), output channel n,
  // so one MMA with N = 3 cout multiplies an input row by the taps of the three
  // output rows it feeds (rows y + 1, y, y - 1 take ky = 0, 1, 2)
  constexpr int kCKB = CIN % 64 == 0 ? 64 : CIN % 32 == 0 ? 32 : 16;
  constexpr int kRB = kCKB * 2, kUnits = kCKB / 8, kChunks = CIN / kCKB;
  for (int i = threadIdx.x; i < 9 * kChunks * cout * kUnits; i += kThreads) {
    const int u = i % kUnits, rest = i / kUnits;
    const int n = rest % cout, blk = rest / cout;  // blk = tap * kChunks + chunk
    const int tap = blk / kChunks, ch = blk - tap * kChunks;
    const int ky = tap / 3, kx = tap - 3 * ky;
    const uint32_t off = (uint32_t)(((kx * kChunks + ch) * 3 * cout + (2 - ky) * cout + n) * kRB +
                                    u * 16);
    *reinterpret_cast<uint4 *>(wsm + swz<kRB>(off)) = *reinterpret_cast<const uint4 *>(
        a.w + (size_t)n * 9 * cin + tap * cin + ch * kCKB + u * 8);
  }
  for (int c = threadIdx.x; c < cout; c += kThreads) s_bias[c] = a.bias ? a.bias[c] : 0.f;
  // generic-proxy stores must be visible to the tensor cores' reads
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *s_tmem;

  if (warp == 0) {
    if (lane == 0) {
      // ------------------------------------------------ TMA producer: input rows
      asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&amap))
                   : "memory");
      uint32_t j = 0, issued = 0, last_par = 0;
      const int chunks = (cin + 63) / 64;
      const uint32_t row_bytes = (uint32_t)chunks * (uint32_t)(kRowPx * 128);
      for (int64_t t = blockIdx.x; t < a.total && !*s_abort; t += gridDim.x) {
        const int sx = (int)(t % a.strips_x);
        const int64_t r = t / a.strips_x;
        const int sy = (int)(r % a.strips_y), b = (int)(r / a.strips_y);
        const int r0 = sy * a.strip_h, r1 = min(r0 + a.strip_h, a.H);
        bool ok = true;
        for (int yi = r0 - 1; yi <= r1; yi++, j++) {
          const int slot = (int)(j % (uint32_t)ns);
          const uint32_t par = (j / (uint32_t)ns) & 1u;
          if (!mbar_wait(&row_empty[slot], par ^ 1u)) {
            atomicOr(a.err, 1);
            *s_abort = 1;
            ok = false;
            break;
          }
          uint8_t *dst = slots + slot * a.slot_bytes;
          mbar_expect_tx(&row_full[slot], row_bytes);
          if (!(j == 0 && __ldg(&g_test_stall)))
            for (int c = 0; c < chunks; c++)
              tma_load_4d(dst + c * kRowChunkBytes, &amap, c * 64, sx * 128 - 1, yi, b,
                          &row_full[slot]);
          issued |= 1u << slot;
          last_par = (last_par & ~(1u << slot)) | (par << slot);
        }
        if (!ok) break;
      }
      for (int s = 0; s < ns; s++)
        if ((issued >> s) & 1u)
          if (!mbar_wait(&row_full[s], (last_par >> s) & 1u)) atomicOr(a.err, 1);
    }
  } else if (warp == 1) {
    {
      // ------------------------------------------------ MMA issuer (whole warp)
      // Input-row stationary: input row yi feeds output rows yi - 1, yi, yi + 1
      // (taps ky = 2, 1, 0), whose accumulators are consecutive blocks of cout
      // columns in a ring of nacc blocks; per (kx, 16-channel step) one MMA with
      // N = 3 cout covers all three (split in two where the ring wraps; fewer
      // rows at a strip's edges).  Each output row still receives its taps in
      // the order ky, kx, channel step.  The first MMA into a block (the row
      // yi + 1 block, at kx = 0 and step 0) overwrites it.
      const uint32_t idesc0 = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(128 >> 4) << 24);
      const uint32_t slots_u = smem_u32(slots);
      constexpr int kCKB = CIN % 64 == 0 ? 64 : CIN % 32 == 0 ? 32 : 16;
      constexpr int kRB = kCKB * 2, kSteps = kCKB / 16, kChunks = CIN / kCKB;
      const uint64_t dw0 = sdesc_swz<kRB>(smem_u32(wsm));
      const uint32_t row16 = (uint32_t)kRB / 16;  // one weight row, 16-byte units
      const uint32_t R = (uint32_t)a.nacc;
      const uint32_t wrow = (uint32_t)cout * row16;  // one block of cout weight rows
      const uint32_t kxblk = 3u * wrow;               // one (kx, chunk) weight block
      // instruction descriptor of n output-row blocks
      auto idesc_n = [&](uint32_t n) { return idesc0 | (((n * (uint32_t)cout) >> 3) << 17); };
      uint32_t j0 = 0, o0 = 0;
      bool ok = true;
      for (int64_t t = blockIdx.x; t < a.total && ok && !__shfl_sync(0xffffffffu, *s_abort, 0);
           t += gridDim.x) {
        const int64_t r = t / a.strips_x;
        const int sy = (int)(r % a.strips_y);
        const int r0 = sy * a.strip_h, r1 = min(r0 + a.strip_h, a.H);
        for (int yi = r0 - 1; yi <= r1 && ok; yi++) {
          const uint32_t jl = j0 + (uint32_t)(yi - r0 + 1);  // load index of input row yi
          ok = __all_sync(0xffffffffu, mbar_wait(&row_full[jl % (uint32_t)ns], (jl / (uint32_t)ns) & 1u));
          const int lo = max(yi - 1, r0), hi = min(yi + 1, r1 - 1);
          const bool fresh = (yi + 1 <= r1 - 1);  // row yi + 1 starts here
          const uint32_t olo = o0 + (uint32_t)(lo - r0), ohi = o0 + (uint32_t)(hi - r0);
          if (ok && fresh)
            ok = __all_sync(0xffffffffu, mbar_wait(&acc_empty[ohi % R], ((ohi / R) & 1u) ^ 1u));
          if (!ok) {
            if (lane == 0) {
              atomicOr(a.err, 1);
              *s_abort = 1;
            }
            break;
          }
          tc_fence_after();
          const uint64_t da = sdesc_sw128(slots_u + (jl % (uint32_t)ns) * (uint32_t)a.slot_bytes);
          // blocks of the rows lo..hi (weight rows from block position p0), split in two
          // where the ring wraps: TMEM column, N and weight offset of both parts as
          // plain scalars, so that the MMAs below take them from uniform registers
          const uint32_t nb = (uint32_t)(hi - lo + 1), p0 = (uint32_t)(lo - yi + 1);
          const uint32_t g = olo % R, n0 = min(nb, R - g), n1 = nb - n0;
          const uint32_t d0 = tmem + g * (uint32_t)cout, i0 = idesc_n(n0), i1 = idesc_n(n1);
          const uint64_t w0 = dw0 + (uint64_t)(p0 * wrow), w1 = dw0 + (uint64_t)((p0 + n0) * wrow);
          if (fresh) {
            // the first MMA of row yi + 1: rows lo..hi - 1 accumulate, row hi starts
            const uint32_t h0 = min(nb - 1u, n0), h1 = nb - 1u - h0;
            if (h0) tc_mma_w(d0, da, w0, idesc_n(h0), 1u);
            if (h1) tc_mma_w(tmem, da, w1, idesc_n(h1), 1u);
            tc_mma_w(tmem + (ohi % R) * (uint32_t)cout, da, dw0 + (uint64_t)((p0 + nb - 1u) * wrow),
                     idesc_n(1u), 0u);
          } else {
            tc_mma_w(d0, da, w0, i0, 1u);
            if (n1) tc_mma_w(tmem, da, w1, i1, 1u);
          }
          auto rest = [&](auto two) {
#pragma unroll
            for (int q = 1; q < 3 * (cin / 16); q++) {
              // 16-channel step st of kx: row chunk st / 4, 32-byte column st % 4;
              // weights: block (kx, st / kSteps), 32-byte column st % kSteps
              const int kx = q / (cin / 16), st = q % (cin / 16);
              const uint64_t a_op =
                  da + (uint64_t)(((st >> 2) * kRowChunkBytes + kx * 128 + (st & 3) * 32) >> 4);
              const uint64_t b_off = (uint64_t)((uint32_t)(kx * kChunks + st / kSteps) * kxblk +
                                                (uint32_t)((st % kSteps) * 2));
              tc_mma_w(d0, a_op, w0 + b_off, i0, 1u);
              if constexpr (decltype(two)::value) tc_mma_w(tmem, a_op, w1 + b_off, i1, 1u);
            }
          };
          if (n1) rest(std::true_type{});
          else rest(std::false_type{});
          tc_commit_w(&row_empty[jl % (uint32_t)ns]);       // input row yi is done
          if (yi - 1 >= r0) tc_commit_w(&acc_full[olo % R]);  // output row yi - 1 is complete
        }
        if (!ok) break;
        j0 += (uint32_t)(r1 - r0) + 2u;
        o0 += (uint32_t)(r1 - r0);
      }
      tc_commit_w(drain);
      if (!mbar_wait(drain, 0)) atomicOr(a.err, 1);
    }
  } else {
    // ---------------------------------------------------- epilogue (warps 2-5)
    const int q = warp & 3;
    const int m = q * 32 + lane;
    int acc = 0, turn = 0;
    uint32_t acc_ph = 0;
    bool stop = false;
    for (int64_t t = blockIdx.x; t < a.total && !stop; t += gridDim.x) {
      const int sx = (int)(t % a.strips_x);
      const int64_t r = t / a.strips_x;
      const int sy = (int)(r % a.strips_y), b = (int)(r / a.strips_y);
      const int r0 = sy * a.strip_h, r1 = min(r0 + a.strip_h, a.H);
      for (int y = r0; y < r1; y++) {
        if (__shfl_sync(0xffffffffu, *s_abort, 0) ||
            !__all_sync(0xffffffffu, mbar_wait(&acc_full[acc], acc_ph))) {
          if (lane == 0) {
            atomicOr(a.err, 1);
            *s_abort = 1;
          }
          stop = true;
          break;
        }
        tc_fence_after();
        const int64_t pix = ((int64_t)b * a.H + y) * a.W + sx * 128 + m;
        const bf16 *mp = a.mask ? a.mask + pix * a.m_cs + a.m_co : nullptr;
        const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(acc * cout);
#pragma unroll 1
        for (int c0 = 0; c0 < cout; c0 += 32, turn ^= 1) {
          uint8_t *so = outs + (BUFS == 2 ? 2 * q + turn : q) * kOutBytes;
          drain32<BUFS - 1>(taddr + (uint32_t)c0, s_bias + c0, mp ? mp + c0 : nullptr, a.relu, so, lane);
          if (lane == 0) tma_store_4d(&ymap, so, c0, sx * 128 + q * 32, y, b);
        }
        tc_fence_before();
        mbar_arrive(&acc_empty[acc]);
        if (++acc == a.nacc) {
          acc = 0;
          acc_ph ^= 1;
        }
      }
    }
    // the staging buffers are read before the CTA may exit
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }

  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(a.cols)
                 : "memory");
}

constexpr int kRowSmemMax = 232448, kRowSmemHalf = 233472 / 2 - 1024;

// resident weights of the row form: 9 taps x cout rows x cin channels
int row_wbytes(const ConvArgs &a) { return 9 * a.cin * a.cout * 2; }

// shared memory of the row form for `slots` input-row buffers and `bufs` staging buffers
// per epilogue warp, with 1 KB to align them
int row_smem(const ConvArgs &a, int slots, int bufs) {
  return row_wbytes(a) + slots * ((a.cin + 63) / 64) * kRowChunkBytes + 4 * bufs * kOutBytes +
         (bufs == 1 ? 0 : kRowTail) + 1024;
}
// One staging buffer where that puts a second CTA on the SM, or the layer on it at all.
int row_bufs(const ConvArgs &a) {
  const int most = row_smem(a, 4, 1) <= kRowSmemHalf ? kRowSmemHalf : kRowSmemMax;
  return row_smem(a, 4, 2) <= most ? 2 : 1;  // 1: 32 -> 64 and 64 -> 32
}

bool make_row_map(const ConvArgs &a, CUtensorMap *map) {
  EncodeTiledFn enc = encode_fn();
  if (!enc) return false;
  std::memset(map, 0, sizeof(*map));
  const cuuint64_t dims[4] = {(cuuint64_t)a.cin, (cuuint64_t)a.W, (cuuint64_t)a.H,
                              (cuuint64_t)a.B};
  const cuuint64_t cs = (cuuint64_t)a.x_cs * 2;
  const cuuint64_t strides[3] = {cs, cs * (cuuint64_t)a.W, cs * (cuuint64_t)a.W * a.H};
  const cuuint32_t box[4] = {64u, (cuuint32_t)kRowPx, 1u, 1u};
  const cuuint32_t estr[4] = {1u, 1u, 1u, 1u};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<bf16 *>(a.x + a.x_co), dims,
             strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
             CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) ==
         CUDA_SUCCESS;
}

// ------------------------------------------------------------ weight gradient
// dw[co][t][ci] += sum_p dy[p][co] x[p + d_t][ci]: nine GEMMs over the pixels that
// read the same dy.  Both operands come from the NHWC tensors by TMA in the MN-major
// (channel-contiguous) 128-byte-swizzled layout, 64 channels wide.  Per 8 x 16 pixel
// block a CTA loads dy once and x as three boxes of 10 x 16 pixels, one per kx and
// zero-filled outside the image: tap ky's operand is the box started 16 ky pixels on,
// a whole number of swizzle atoms.  M = 128 holds two taps of 64 input channels each
// (the descriptor's stride between channel atoms reaches from one tap's operand to
// the other's), N = up to 64 output channels, K = 16 pixels: five MMAs per step for
// nine taps, into five tensor-memory accumulators.  The pixel blocks are split over
// CTAs, which add their sums to dw.
//
// A CTA has the taps of one kx where those CTAs are all resident.  Bound by the operands' shared-memory reads (6 KB, 48 clocks per MMA whose
// math takes 32) and the issue of MMAs that short (70 clocks).  One tap per CTA, M = 128
// output channels, read dy and x from L2 once per tap and was bound by that: 64 -> 64 at
// 2 x 1024 x 1024 830 us, now 283; 32 -> 32 at 4 x 512 x 512 422 and 134, 192 -> 64 at
// 2 x 512 x 512 448 and 216, 128 -> 128 at 4 x 256 x 256 129 and 88.  From 64 pixel blocks
// on no layer is slower; images of 4096 pixels and less with 128 channels or more, one
// block to a CTA, are by up to 1.7 us (256 -> 256 at 16 x 32 8.1 against 6.4).
struct WgTcArgs {
  float *dw;
  int cin, cout;
  int bx, by;
  int64_t nblk;  // B * by * bx pixel blocks
  int ci_tiles, ksplit;
  int n;         // MMA N: output channels of a tile, a multiple of 16, at most 64
  int *err;
};

// MN-major 128-byte-swizzled descriptor: 8-row K groups 1024 B apart, MN atoms
// of 64 channels `lbo` bytes apart
__device__ __forceinline__ uint64_t sdesc_mn128(uint32_t addr, uint32_t lbo) {
  return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
         ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}

// 4 x 4 transpose among four neighbouring lanes: lane r of them gives v[c] as element
// (r, c) and has element (c, r) as v[c] after.
__device__ __forceinline__ void transpose4(float (&v)[4], int lane) {
  const bool r0 = lane & 1, r1 = lane & 2;
  float t = __shfl_xor_sync(0xffffffffu, r0 ? v[0] : v[1], 1);
  (r0 ? v[0] : v[1]) = t;
  t = __shfl_xor_sync(0xffffffffu, r0 ? v[2] : v[3], 1);
  (r0 ? v[2] : v[3]) = t;
  t = __shfl_xor_sync(0xffffffffu, r1 ? v[0] : v[2], 2);
  (r1 ? v[0] : v[2]) = t;
  t = __shfl_xor_sync(0xffffffffu, r1 ? v[1] : v[3], 2);
  (r1 ? v[1] : v[3]) = t;
}

constexpr int kWgRow = 16 * 128;          // 16 pixels x 64 channels x 2 B
constexpr int kWgBox = 10 * kWgRow;       // one kx: rows -1 .. 8
// G = 1: a CTA has all nine taps; G = 3: those of one kx
template <int G> struct WgCfg {
  static constexpr int kBoxes = 3 / G, kAcc = G == 1 ? 5 : 2, kStages = G == 1 ? 2 : 3;
  static constexpr uint32_t kCols = G == 1 ? 512 : 128;
  static constexpr int kStage = kBoxes * kWgBox + 8 * kWgRow;  // x boxes, then dy
  static constexpr int kSmem = kStages * kStage + 256 + 1024;  // + barriers, alignment slack
  // tap (3 ky + kx) of the lower or upper half of an accumulator
  static __device__ __forceinline__ int tap(int acc, int half, int kx) {
    if (G == 3) return acc == 0 ? 3 * half + kx : half == 0 ? 6 + kx : -1;
    return acc < 3 ? 3 * half + acc : acc == 3 ? 6 + half : half == 0 ? 8 : -1;
  }
};

template <int G>
__global__ void __launch_bounds__(kThreads, 1)
    wgrad_tc_kernel(const __grid_constant__ CUtensorMap dymap,
                    const __grid_constant__ CUtensorMap xmap, WgTcArgs a) {
  using C = WgCfg<G>;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t pad = (1024u - (smem_u32(smem_raw) & 1023u)) & 1023u;
  uint8_t *base = smem_raw + pad;
  // a stage is filled in two parts: dy and the boxes of kx 0 and 1 (or of the one kx),
  // then that of kx 2
  uint64_t *full = reinterpret_cast<uint64_t *>(base + C::kStages * C::kStage);  // [stage][part]
  uint64_t *empty = full + 2 * C::kStages;
  uint64_t *done = empty + C::kStages;
  uint64_t *drain = done + 1;
  uint32_t *s_tmem = reinterpret_cast<uint32_t *>(drain + 1);
  volatile int *s_abort = reinterpret_cast<volatile int *>(s_tmem + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // work item: (co tile, ci tile, K split, kx where a CTA has one)
  int w = (int)blockIdx.x;
  const int kx0 = w % G;
  w /= G;
  const int ks = w % a.ksplit;
  w /= a.ksplit;
  const int cit = w % a.ci_tiles, cot = w / a.ci_tiles;
  const int64_t b0 = a.nblk * ks / a.ksplit, b1 = a.nblk * (ks + 1) / a.ksplit;

  if (threadIdx.x == 0) {
    for (int s = 0; s < 2 * C::kStages; s++) mbar_init(&full[s], 1);
    for (int s = 0; s < C::kStages; s++) mbar_init(&empty[s], 1);
    mbar_init(done, 1);
    mbar_init(drain, 1);
    *s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(s_tmem)),
                 "r"(C::kCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *s_tmem;

  if (warp == 0) {
    if (lane == 0) {
      // ------------------------------------------------ TMA producer
      asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&dymap))
                   : "memory");
      asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&xmap))
                   : "memory");
      int stage = 0;
      uint32_t ph = 0, issued = 0, last_par = 0;
      bool ok = true;
      for (int64_t blk = b0; blk < b1 && ok; blk++) {
        const int tx = (int)(blk % a.bx);
        const int64_t r = blk / a.bx;
        const int ty = (int)(r % a.by), b = (int)(r / a.by);
        uint8_t *sx = base + stage * C::kStage, *sd = sx + C::kBoxes * kWgBox;
        const bool stall = blk == b0 && __ldg(&g_test_stall);
        auto box = [&](int kx, uint64_t *bar) {
          tma_load_4d(sx + kx * kWgBox, &xmap, cit * 64, tx * 16 + kx0 + kx - 1, ty * 8 - 1, b, bar);
        };
        ok = mbar_wait(&empty[stage], ph ^ 1);
        if (!ok) {
          atomicOr(a.err, 1);
          *s_abort = 1;
          break;
        }
        mbar_expect_tx(&full[2 * stage], (uint32_t)((G == 1 ? 2 : 1) * kWgBox + 8 * kWgRow));
        if (G == 1) mbar_expect_tx(&full[2 * stage + 1], (uint32_t)kWgBox);
        if (!stall) {
          tma_load_4d(sd, &dymap, cot * a.n, tx * 16, ty * 8, b, &full[2 * stage]);
          box(0, &full[2 * stage]);
          if (G == 1) {
            box(1, &full[2 * stage]);
            box(2, &full[2 * stage + 1]);
          }
        }
        issued |= 1u << stage;
        last_par = (last_par & ~(1u << stage)) | (ph << stage);
        if (++stage == C::kStages) {
          stage = 0;
          ph ^= 1;
        }
      }
      for (int s = 0; s < C::kStages; s++)
        if ((issued >> s) & 1u)
          for (int part = 0; part < (G == 1 ? 2 : 1); part++)
            if (!mbar_wait(&full[2 * s + part], (last_par >> s) & 1u)) atomicOr(a.err, 1);
    }
  } else if (warp == 1) {
    {
      // ------------------------------------------------ MMA issuer (whole warp)
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) |
                             ((uint32_t)(a.n >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
      int stage = 0;
      uint32_t ph = 0, more = 0;
      for (int64_t blk = b0; blk < b1 && !__shfl_sync(0xffffffffu, *s_abort, 0); blk++) {
        const uint32_t sx = smem_u32(base + stage * C::kStage);
        const uint64_t db = sdesc_mn128(sx + C::kBoxes * kWgBox, kWgRow);
        auto row = [&](int acc, int k, uint64_t da) {  // pixel row k of the block
          tc_mma_w(tmem + (uint32_t)(64 * acc), da + (uint64_t)(k * (kWgRow >> 4)),
                 db + (uint64_t)(k * (kWgRow >> 4)), idesc, more | (uint32_t)k);
        };
        bool ok = __all_sync(0xffffffffu, mbar_wait(&full[2 * stage], ph));
        if (ok) {
          tc_fence_after();
          if constexpr (G == 3) {
#pragma unroll
            for (int k = 0; k < 8; k++) {
              row(0, k, sdesc_mn128(sx, kWgRow));                 // ky 0, 1
              row(1, k, sdesc_mn128(sx + 2 * kWgRow, kWgRow));    // ky 2 (lower half)
            }
          } else {
#pragma unroll
            for (int k = 0; k < 8; k++) {
              row(0, k, sdesc_mn128(sx, kWgRow));                 // ky 0, 1 of kx 0
              row(1, k, sdesc_mn128(sx + kWgBox, kWgRow));        // ky 0, 1 of kx 1
              row(3, k, sdesc_mn128(sx + 2 * kWgRow, kWgBox));    // ky 2 of kx 0, 1
            }
            ok = __all_sync(0xffffffffu, mbar_wait(&full[2 * stage + 1], ph));
          }
        }
        if (!ok) {
          if (lane == 0) {
            atomicOr(a.err, 1);
            *s_abort = 1;
          }
          break;
        }
        tc_fence_after();
        // ky 0, 1 of kx 2; ky 2 of kx 2, whose upper half (the rows below, or dy's
        // first) is not used
        if constexpr (G == 1) {
#pragma unroll
          for (int k = 0; k < 8; k++) {
            row(2, k, sdesc_mn128(sx + 2 * kWgBox, kWgRow));
            row(4, k, sdesc_mn128(sx + 2 * kWgBox + 2 * kWgRow, kWgRow));
          }
        }
        tc_commit_w(&empty[stage]);
        more = 1;
        if (++stage == C::kStages) {
          stage = 0;
          ph ^= 1;
        }
      }
      tc_commit_w(done);
      tc_commit_w(drain);
      if (!mbar_wait(drain, 0)) atomicOr(a.err, 1);
    }
  } else {
    // ---------------------------------------------------- epilogue (warps 2-5)
    const int q = warp & 3, row = q * 32 + lane;
    const bool ok = __all_sync(0xffffffffu, mbar_wait(done, 0));
    if (!ok && lane == 0) {
      atomicOr(a.err, 1);
      *s_abort = 1;
    }
    if (ok && b1 > b0 && !__shfl_sync(0xffffffffu, *s_abort, 0)) {
      tc_fence_after();
      // row (half, ci) of every accumulator.  Four lanes exchange 4 x 4 blocks, so that each
      // adds 16 bytes: four input channels of one output channel, eight such lanes side
      // by side (dw and rows of 16 channels and more are 16-byte aligned).  4-byte adds
      // took 17.1 us for one pixel block and 64 x 64 channels in one CTA, these 11.6.
      const int half = row >> 6, ci = cit * 64 + (row & 60);
#pragma unroll 1
      for (int acc = 0; acc < C::kAcc; acc++) {
        const int tap = C::tap(acc, half, kx0);
#pragma unroll 1
        for (int c0 = 0; c0 < a.n; c0 += 32) {
          // two 16-column loads in flight; the second is not used by a tile of 16 or 48
          uint32_t rr[2][16];
          const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(64 * acc + c0);
          tmem_ld16(taddr, rr[0]);
          tmem_ld16(taddr + 16u, rr[1]);
          tmem_wait_ld();
          float *o = a.dw + ((int64_t)(cot * a.n + c0 + (lane & 3)) * 9 + tap) * a.cin + ci;
          const int left = tap >= 0 && ci < a.cin
                               ? min(a.n - c0, a.cout - cot * a.n - c0) - (lane & 3) : 0;
#pragma unroll
          for (int c = 0; c < 32; c += 4) {
            float v[4];
#pragma unroll
            for (int j = 0; j < 4; j++) v[j] = __uint_as_float(rr[c >> 4][(c & 15) + j]);
            transpose4(v, lane);
            if (c < left)
              atomicAdd(reinterpret_cast<float4 *>(o + (int64_t)c * 9 * a.cin),
                        make_float4(v[0], v[1], v[2], v[3]));
          }
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(C::kCols)
                 : "memory");
}

bool make_nhwc_map(const __nv_bfloat16 *p, int cs, int co, int C, int W, int H, int B, int rows,
                   CUtensorMap *map) {
  EncodeTiledFn enc = encode_fn();
  if (!enc) return false;
  std::memset(map, 0, sizeof(*map));
  const cuuint64_t dims[4] = {(cuuint64_t)C, (cuuint64_t)W, (cuuint64_t)H, (cuuint64_t)B};
  const cuuint64_t s0 = (cuuint64_t)cs * 2;
  const cuuint64_t strides[3] = {s0, s0 * (cuuint64_t)W, s0 * (cuuint64_t)W * H};
  const cuuint32_t box[4] = {64u, 16u, (cuuint32_t)rows, 1u};
  const cuuint32_t estr[4] = {1u, 1u, 1u, 1u};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<__nv_bfloat16 *>(p + co), dims,
             strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
             CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) ==
         CUDA_SUCCESS;
}

template <int G>
cudaError_t launch_wgrad(const CUtensorMap &dymap, const CUtensorMap &xmap, const WgTcArgs &w,
                         int tiles, cudaStream_t st) {
  constexpr int smem = WgCfg<G>::kSmem;
  const cudaError_t e =
      cudaFuncSetAttribute(wgrad_tc_kernel<G>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  wgrad_tc_kernel<G><<<(unsigned)(tiles * w.ksplit * G), kThreads, smem, st>>>(dymap, xmap, w);
  return cudaGetLastError();
}

}  // namespace

int conv_tc_chunk(int cin) {
  return cin % 64 == 0 ? 64 : cin % 32 == 0 ? 32 : cin == 16 ? 16 : 0;
}

int conv_tc_ntile(int cout) {
  if (cout <= 128) return (cout % 32 == 0) ? cout : 0;
  if (cout % 128 == 0) return 128;
  if (cout % 96 == 0) return 96;
  if (cout % 64 == 0) return 64;
  return cout % 32 == 0 ? 32 : 0;
}

bool conv_row_ok(const ConvArgs &a) {
  return conv_tc_ok(a) && a.W % 128 == 0 &&
         (a.cin == 16 || a.cin == 32 || a.cin == 64 || a.cin == 96 || a.cin == 128) &&
         a.cout % 32 == 0 &&
         a.cout <= kRowMaxCout && row_wbytes(a) <= 112 * 1024 && row_smem(a, 4, 1) <= kRowSmemMax;
}

cudaError_t launch_conv3x3_row(const ConvArgs &a, cudaStream_t st) {
  if (!conv_row_ok(a)) return cudaErrorInvalidValue;
  CUtensorMap amap, ymap;
  if (!make_row_map(a, &amap) || !make_out_map(a, 32, 1, &ymap)) return cudaErrorInvalidValue;
  RowArgs r{};
  r.mask = a.mask;
  r.m_cs = a.m_cs;
  r.m_co = a.m_co;
  r.bias = a.bias;
  r.w = a.w;
  r.cin = a.cin;
  r.cout = a.cout;
  r.relu = a.relu;
  r.H = a.H;
  r.W = a.W;
  // half of tensor memory for each of two CTAs per SM, all of it for one
  const int bufs = row_bufs(a);
  r.cols = row_smem(a, 4, bufs) <= kRowSmemHalf ? 256u : 512u;
  r.nacc = std::min<int>(kMaxAcc, (int)r.cols / a.cout);
  r.wbytes = row_wbytes(a);
  r.slot_bytes = ((a.cin + 63) / 64) * kRowChunkBytes;
  // two CTAs per SM where four input rows fit beside the weights, else one
  const int most = r.cols == 256u ? kRowSmemHalf : kRowSmemMax;
  int slots = kRowMaxSlots;
  while (slots > 4 && row_smem(a, slots, bufs) > most) slots--;
  r.nslots = slots;
  cudaError_t e = err_word(&r.err);
  if (e != cudaSuccess) return e;
  const int per_sm = 512 / (int)r.cols;
  const int smem = std::max(row_smem(a, slots, bufs), 232448 / (per_sm + 1) + 1024);
  auto kern = a.cin == 16   ? conv_row_kernel<16, 2>
              : a.cin == 32 ? (bufs == 1 ? conv_row_kernel<32, 1> : conv_row_kernel<32, 2>)
              : a.cin == 64 ? (bufs == 1 ? conv_row_kernel<64, 1> : conv_row_kernel<64, 2>)
              : a.cin == 96 ? conv_row_kernel<96, 2>
                            : conv_row_kernel<128, 2>;
  e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout,
                           (int)cudaSharedmemCarveoutMaxShared);
  if (e != cudaSuccess) return e;
  const int occ = occupancy(kern, smem, per_sm);
  const int64_t ctas = (int64_t)sm_count() * occ;
  r.strips_x = a.W / 128;
  // strips of up to 32 rows; shorter where that leaves too few strips per CTA
  int sh = std::min(32, a.H);
  while (sh > 8 && (int64_t)a.B * r.strips_x * ((a.H + sh - 1) / sh) < 4 * ctas) sh /= 2;
  r.strip_h = sh;
  r.strips_y = (a.H + sh - 1) / sh;
  r.total = (int64_t)a.B * r.strips_y * r.strips_x;
  const int64_t grid = std::min<int64_t>(r.total, ctas);
  kern<<<(unsigned)grid, kThreads, smem, st>>>(amap, ymap, r);
  return cudaGetLastError();
}

bool conv_tc_ok(const ConvArgs &a) {
  return conv_shape_ok(a) && conv_tc_chunk(a.cin) != 0 && conv_tc_ntile(a.cout) != 0 &&
         a.y_cs % 8 == 0 && a.y_co % 8 == 0 && (!a.mask || (a.m_cs % 8 == 0 && a.m_co % 8 == 0)) &&
         a.cin <= 65535 && a.cout <= kMaxCout;
}

cudaError_t launch_conv3x3_tc(const ConvArgs &a, cudaStream_t st) {
  if (!conv_tc_ok(a)) return cudaErrorInvalidValue;
  if (conv_row_ok(a)) return launch_conv3x3_row(a, st);
  const int ck = conv_tc_chunk(a.cin), nt = conv_tc_ntile(a.cout);
  if (ck == 64) return launch_ck<64>(a, nt, st);
  if (ck == 32) return launch_ck<32>(a, nt, st);
  return launch_ck<16>(a, nt, st);
}

bool wgrad_tc_ok(const WgradArgs &a) {
  return a.B >= 1 && a.H >= 8 && a.W >= 16 && a.H % 8 == 0 && a.W % 16 == 0 && a.cin % 16 == 0 &&
         a.cout % 16 == 0 && a.x_cs % 8 == 0 && a.x_co % 8 == 0 && a.dy_cs % 8 == 0 &&
         a.dy_co % 8 == 0 && a.x_co + a.cin <= a.x_cs && a.dy_co + a.cout <= a.dy_cs &&
         (reinterpret_cast<uintptr_t>(a.dw) & 15) == 0;
}

cudaError_t launch_conv3x3_wgrad_tc(const WgradArgs &a, cudaStream_t st) {
  if (!wgrad_tc_ok(a)) return cudaErrorInvalidValue;
  CUtensorMap dymap, xmap;
  if (!make_nhwc_map(a.dy, a.dy_cs, a.dy_co, a.cout, a.W, a.H, a.B, 8, &dymap) ||
      !make_nhwc_map(a.x, a.x_cs, a.x_co, a.cin, a.W, a.H, a.B, 10, &xmap))
    return cudaErrorInvalidValue;
  WgTcArgs w{};
  w.dw = a.dw;
  w.cin = a.cin;
  w.cout = a.cout;
  w.bx = a.W / 16;
  w.by = a.H / 8;
  w.nblk = (int64_t)a.B * w.by * w.bx;
  w.ci_tiles = (a.cin + 63) / 64;
  int tiles = w.ci_tiles * ((a.cout + 63) / 64);
  // K splits: as many as fill the device twice with tiles of 128 output channels x 64 or
  // 128 input channels x one tap.  The tensor cores' accumulation truncates, so the
  // split decides the result to 1e-4 of it, and stays where it was when a CTA had one
  // such tile.
  const int64_t cols = 9LL * ((a.cout + 127) / 128) * (a.cin > 64 ? (a.cin + 127) / 128 : 1);
  w.ksplit = (int)std::max<int64_t>(1, std::min<int64_t>(w.nblk, (2LL * sm_count() + cols - 1) / cols));
  cudaError_t e = err_word(&w.err);
  if (e != cudaSuccess) return e;
  // A CTA per kx where all of them are resident at once, two to an SM (64 -> 128 at
  // 64 x 64, 64 nine-tap CTAs: 8.1 against 11.7 us; 128 -> 128 at 128 x 128, 132: 17.8 and
  // 15.9), and 32 output channels each where those are still resident and have few pixel
  // blocks, so that adding them up is most of the time (64 -> 64 at 32 x 32 5.4 against
  // 6.7 us, at 128 x 128 8.6 both ways).
  const bool three = 3 * tiles * w.ksplit <= 2 * sm_count();
  const bool half = three && 6 * tiles * w.ksplit <= 2 * sm_count() && w.nblk <= 4 * w.ksplit;
  w.n = std::min(half ? 32 : 64, a.cout);
  tiles = w.ci_tiles * ((a.cout + w.n - 1) / w.n);
  return three ? launch_wgrad<3>(dymap, xmap, w, tiles, st) : launch_wgrad<1>(dymap, xmap, w, tiles, st);
}

int conv_tc_error() {
  std::lock_guard<std::mutex> l(g_err_mutex);
  return g_err_host ? *(volatile int *)g_err_host : 0;
}

void conv_tc_clear_error() {
  std::lock_guard<std::mutex> l(g_err_mutex);
  if (g_err_host) *(volatile int *)g_err_host = 0;
}

}  // namespace ctas

// Test aid of the C ABI (ctas_learned.h): arm or disarm the stall of the
// tcgen05 convolution kernels on the current device.
extern "C" int ctas_nn_test_timeout(int32_t enable) {
  const int stall = enable ? 1 : 0;
  const uint32_t limit = enable ? (1u << 12) : ctas::kWaitLimit;
  if (cudaMemcpyToSymbol(ctas::g_test_stall, &stall, sizeof(stall)) != cudaSuccess ||
      cudaMemcpyToSymbol(ctas::g_wait_limit, &limit, sizeof(limit)) != cudaSuccess) {
    cudaGetLastError();
    return CTAS_E_CUDA;
  }
  return CTAS_OK;
}
