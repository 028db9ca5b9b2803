// Device-side building blocks of the tcgen05 GEMMs (sm_103a): split-plane element types,
// mbarrier / TMA / tcgen05 inline PTX and the bounded waits.  Shared by the dense-embedding
// persistent GEMM (gemm_tc.cu) and the grouped sector-block GEMM (grouped.cu).
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "gb_common.h"

namespace gb {

// bound on the waits of a kernel's drain path (copies already issued, MMAs already
// committed): those always complete, so this bound only guards against a broken pipeline
constexpr unsigned long long DRAIN_WAIT_NS = 2000000000ull;

// ------------------------------------------------------------------ plane element types
// BF16 planes (bf16x3) or TF32 values in 32-bit words (tf32x3).  A k-block is one 128-byte
// swizzle row: 64 BF16 or 32 TF32 elements.
template <typename E>
constexpr int bk_of() {
  return 128 / (int)sizeof(E);
}
__device__ __forceinline__ float tf32_rna(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return __uint_as_float(r);
}
// hi/lo split of a value rounded to FP32: its 24 bits hold the 16 (BF16) or 22 (TF32) bits
// the two planes keep, and the split needs no FP64 arithmetic (GB300's FP64 rate is a small
// fraction of its FP32 rate)
__device__ __forceinline__ void split_put_f(__nv_bfloat16* hi, __nv_bfloat16* lo, int64_t i,
                                            float v) {
  const __nv_bfloat16 h = __float2bfloat16_rn(v);
  hi[i] = h;
  lo[i] = __float2bfloat16_rn(v - __bfloat162float(h));
}
__device__ __forceinline__ void split_put_f(float* hi, float* lo, int64_t i, float v) {
  const float h = tf32_rna(v);
  hi[i] = h;
  lo[i] = tf32_rna(v - h);
}
__device__ __forceinline__ bool plane_nz(__nv_bfloat16 a) { return __bfloat162float(a) != 0.f; }
__device__ __forceinline__ bool plane_nz(float a) { return a != 0.f; }
inline bool is_tf32(int prec) { return prec == GB_PREC_TF32X3; }

// ------------------------------------------------------------------ FP32 <-> FP64 by the bits
// Conversions run on the FP64 pipe (one warp instruction per 16 clocks and SM); these give the
// same results with a handful of integer instructions.
// (double)x; subnormal and non-finite values take the conversion
__device__ __forceinline__ double to_double(float x) {
  const uint32_t u = __float_as_uint(x), mag = u & 0x7fffffffu;
  if (__builtin_expect(mag - 0x00800000u < 0x7f000000u, 1))
    return __hiloint2double((int)((u & 0x80000000u) | ((mag >> 3) + 0x38000000u)),
                            (int)(u << 29));
  return mag ? (double)x : __hiloint2double((int)u, 0);
}
__device__ __forceinline__ double to_double(double x) { return x; }
// (float)x, to nearest even, without the FP64 pipe; values outside FP32's normal range (and
// their rounding) take the conversion
__device__ __forceinline__ float to_float(double x) {
  const uint32_t hi = (uint32_t)__double2hiint(x), lo = (uint32_t)__double2loint(x);
  const uint32_t mag = hi & 0x7fffffffu;
  if (__builtin_expect(mag - 0x38100000u < 0x0fd00000u, 1)) {
    // 20 + 3 bits kept; the rest decides
    uint32_t r = ((mag - 0x38000000u) << 3) | (lo >> 29);
    const uint32_t rest = lo & 0x1fffffffu;
    r += (rest > 0x10000000u || (rest == 0x10000000u && (r & 1u))) ? 1u : 0u;
    return __uint_as_float((hi & 0x80000000u) | r);
  }
  return (mag | lo) ? (float)x : __uint_as_float(hi & 0x80000000u);
}

// ------------------------------------------------------------------ PTX helpers
// Programmatic dependent launch: kernels of a chain start while the one before them drains
// (launch_chained), set themselves up and wait here for its memory before they touch any of it.
// Every thread waits, so a kernel's end implies its predecessors' ends.  Data that the kernel
// before may have written is read through plain pointers: a load through a const __restrict__
// one may be moved above the wait.  Measured: an apply of two 128 x 256 x 256 complex products
// (four launches) 41.5 us in plain launches, 34.0 us chained; a D = 32 time step of 3900 launches
// 40.2 and 32.5 ms.
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// the next kernel of the chain may start (once every CTA of this one has started)
__device__ __forceinline__ void chain_release() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ unsigned long long globaltimer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
               : "memory");
}
// The warp's index as a value the compiler knows to be the same in all lanes, and one lane of a
// converged warp, known to be a single one.  Copies, MMAs and commits take their operands from
// uniform registers: under a plain `lane == 0` each of them is issued in a loop over whatever
// lanes may be active, and the issuing threads, not the memory or the tensor cores, set the pace
// (a wait, an expect and a copy: 302 clocks under `lane == 0`, 191 here).
__device__ __forceinline__ int warp_index() {
  return __shfl_sync(0xffffffffu, (int)threadIdx.x / 32, 0);
}
__device__ __forceinline__ bool elect_one() {
  uint32_t one;
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b32 r;\n\t"
      "elect.sync r|p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(one));
  return one != 0;
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// bounded wait: returns false (and records a timeout) when the bound expires
__device__ __forceinline__ bool mbar_wait_bounded(uint32_t bar, uint32_t parity, int* status,
                                                  unsigned long long bound_ns) {
  if (mbar_try_wait(bar, parity)) return true;
  unsigned long long t0 = globaltimer();
  while (!mbar_try_wait(bar, parity)) {
    if (globaltimer() - t0 > bound_ns) {
      atomicExch(status, GB_ERR_TIMEOUT);
      return false;
    }
  }
  return true;
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, uint32_t bar,
                                            int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(dst),
      "l"((unsigned long long)map), "r"(bar), "r"(x), "r"(y), "r"(z)
      : "memory");
}
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFF);        // start address
  d |= (uint64_t)1 << 16;                        // leading byte offset (unused for SW128 K-major)
  d |= (uint64_t)(1024 >> 4) << 32;              // stride byte offset: 8 rows x 128 B
  d |= (uint64_t)1 << 46;                        // descriptor version (sm_100 family)
  d |= (uint64_t)2 << 61;                        // 128-byte swizzle
  return d;
}
// kind::f16 instruction descriptor: BF16 x BF16 -> F32, both K-major
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) |
         ((uint32_t)(M >> 4) << 24);
}
__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc,
                                         uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate));
}
// kind::tf32 instruction descriptor: TF32 x TF32 -> F32, both K-major
__host__ __device__ constexpr uint32_t idesc_tf32(int M, int N) {
  return (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(N >> 3) << 17) |
         ((uint32_t)(M >> 4) << 24);
}
__device__ __forceinline__ void mma_tf32(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc,
                                         uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate));
}
__device__ __forceinline__ void mma_commit(uint32_t bar) {
  asm volatile(
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
      : "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

#define TMEM_LD32(taddr, r)                                                                   \
  asm volatile(                                                                               \
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13," \
      "%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"      \
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),  \
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),           \
        "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),        \
        "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),        \
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]),        \
        "=r"(r[31])                                                                           \
      : "r"(taddr))
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

// ------------------------------------------------------------------ tile counter
// counter[0] hands out tiles, counter[1] counts the CTAs that are done with it: the last one
// leaves both at zero for the next launch (a memset in between would cost a launch and break
// the chain of launches).  Call from one thread, after the CTA's last tile.
__device__ __forceinline__ void tiles_done(unsigned int* counter) {
  if (atomicAdd(&counter[1], 1u) == gridDim.x - 1) {
    counter[0] = 0;
    counter[1] = 0;
    __threadfence();
  }
}

}  // namespace gb
