// bp_stage.cuh -- device helpers shared by the staged backprojection kernels:
// mbarriers with bounded waits, asynchronous copies, packed float arithmetic with
// explicit rounding, and the start of a tile's detector window.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdint>

namespace ctas {
namespace {

constexpr uint32_t kWaitLimit = 1u << 22;
constexpr float kMagic = 12582912.0f;  // 1.5 * 2^23
constexpr uint32_t kMagicBits = 0x4B400000u;
constexpr float kTwoM22 = 2.384185791015625e-07f;  // 2^-22

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(unsigned long long *bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count)
               : "memory");
}

__device__ __forceinline__ void mbar_inval(unsigned long long *bar) {
  asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void mbar_arrive(unsigned long long *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(unsigned long long *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(unsigned long long *bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// bounded wait: false when the limit ran out
__device__ __forceinline__ bool mbar_wait(unsigned long long *bar, uint32_t parity,
                                          uint32_t limit = kWaitLimit) {
  for (uint32_t it = 0; it < limit; ++it)
    if (mbar_try_wait(bar, parity)) return true;
  return false;
}

__device__ __forceinline__ void tma_load_row(void *dst, const CUtensorMap *map, int x, int y,
                                             unsigned long long *bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3}], [%4];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(smem_u32(bar))
      : "memory");
}

// Untiled copy of `bytes` (a multiple of 16) between 16-byte boundaries.
__device__ __forceinline__ void bulk_load(void *dst, const void *src, uint32_t bytes,
                                          unsigned long long *bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(src)), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}

// packed f32x2 adds (sm_100a), explicit rounding; inputs never come straight
// from a multiply (a packed multiply-add chain may be fused)
__device__ __forceinline__ float2 add2_rn(float2 a, float2 b) {
  float2 r;
  asm("{\n .reg .b64 ra, rb, rr;\n mov.b64 ra, {%2, %3};\n mov.b64 rb, {%4, %5};\n"
      " add.rn.f32x2 rr, ra, rb;\n mov.b64 {%0, %1}, rr;\n}\n"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return r;
}
__device__ __forceinline__ float2 add2_rm(float2 a, float2 b) {
  float2 r;
  asm("{\n .reg .b64 ra, rb, rr;\n mov.b64 ra, {%2, %3};\n mov.b64 rb, {%4, %5};\n"
      " add.rm.f32x2 rr, ra, rb;\n mov.b64 {%0, %1}, rr;\n}\n"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return r;
}

__device__ __forceinline__ float2 add2_rp(float2 a, float2 b) {
  float2 r;
  asm("{\n .reg .b64 ra, rb, rr;\n mov.b64 ra, {%2, %3};\n mov.b64 rb, {%4, %5};\n"
      " add.rp.f32x2 rr, ra, rb;\n mov.b64 {%0, %1}, rr;\n}\n"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return r;
}

// Packed product a * b formed as fma(a, b, +0): one rounding, like a
// multiply, but the compiler cannot contract it into a following add (a
// packed multiply with explicit rounding does get contracted).  It differs
// from the product only in the sign of a zero result, which changes no
// floor index downstream.
__device__ __forceinline__ float2 mul2z_rn(float2 a, float2 b) {
  float2 r;
  asm("{\n .reg .b64 ra, rb, rz, rr;\n mov.b64 ra, {%2, %3};\n mov.b64 rb, {%4, %5};\n"
      " mov.b64 rz, 0;\n fma.rn.f32x2 rr, ra, rb, rz;\n mov.b64 {%0, %1}, rr;\n}\n"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return r;
}

__device__ __forceinline__ float2 fma2_rn(float2 a, float2 b, float2 c) {
  float2 r;
  asm("{\n .reg .b64 ra, rb, rc, rr;\n mov.b64 ra, {%2, %3};\n mov.b64 rb, {%4, %5};\n"
      " mov.b64 rc, {%6, %7};\n fma.rn.f32x2 rr, ra, rb, rc;\n mov.b64 {%0, %1}, rr;\n}\n"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return r;
}

// x << 2 as a funnel shift of (x : lo) with lo < 2^30, so that it runs on the
// integer ALU rather than as a multiply-add
__device__ __forceinline__ uint32_t shl2_alu(uint32_t x, uint32_t lo) {
  uint32_t r;
  asm("shf.l.wrap.b32 %0, %1, %2, 2;" : "=r"(r) : "r"(lo), "r"(x));
  return r;
}

// Shared loads of a released stage.  Not volatile: the address depends on
// parameters read after the stage's barrier wait, which orders the load.
__device__ __forceinline__ float lds_f32(uint32_t addr) {
  float v;
  asm("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr));
  return v;
}

__device__ __forceinline__ float2 lds_f32x2(uint32_t addr) {
  float2 v;
  asm("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(addr));
  return v;
}

// Lowest detector index any pixel of the tile can reach, minus a margin,
// rounded down to a multiple of `align` elements (16-byte TMA alignment).
// (ja, jb), (ia, ib): reference coordinates of the tile's first and last
// rows and columns; the index is affine in them, so its minimum is at a
// corner (rounding moves it by far less than the margin).
__device__ __forceinline__ int window_start_trunc(float sx, float cy, float base, float ja,
                                                  float jb, float ia, float ib, float c,
                                                  int align, float *tmin_out = nullptr) {
  const float jc0 = __fsub_rn(ja, c), jc1 = __fsub_rn(jb, c);
  const float d0 = __fmul_rn(cy, ia), d1 = __fmul_rn(cy, ib);
  const float b0 = __fadd_rn(base, __fmul_rn(sx, jc0)), b1 = __fadd_rn(base, __fmul_rn(sx, jc1));
  const float tmin = fminf(fminf(__fadd_rn(b0, d0), __fadd_rn(b0, d1)),
                           fminf(__fadd_rn(b1, d0), __fadd_rn(b1, d1)));
  if (tmin_out) *tmin_out = tmin;
  const int lo = (int)floorf(tmin) - 2;
  return lo & ~(align - 1);
}

__device__ __forceinline__ int window_start_linear(float sx, float cy, float t0, float ja,
                                                   float jb, float ia, float ib, int align) {
  const float a = fmaf(sx, ja, t0), b = fmaf(sx, jb, t0);
  const float tmin = fminf(fminf(fmaf(cy, ia, a), fmaf(cy, ib, a)),
                           fminf(fmaf(cy, ia, b), fmaf(cy, ib, b)));
  const int lo = (int)floorf(tmin) - 2;
  return lo & ~(align - 1);
}

}  // namespace
}  // namespace ctas
