// Building blocks of the tensor-core kernels: tcgen05 (fp16 operands, fp32
// accumulators in tensor memory), mbarriers, the split of fp32 values into
// two fp16 parts, vector reductions.
//
// Operands lie in shared memory as K-major core matrices without swizzle: 8
// rows (of M or N) x 16 bytes (8 samples), 128 contiguous bytes.  The core
// matrix of row group r and sample octet o sits at r * 128 + o * lbo.
#pragma once

#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace gbn {
namespace tc {

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void bar_init(uint64_t* bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void bar_init_fence() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// Waits for the completion of the barrier's phase `parity`.  Gives up after
// about a second of clock cycles: *err is set and false returned.
__device__ __forceinline__ bool bar_wait(uint64_t* bar, uint32_t parity, int* err) {
  const long long t0 = clock64();
  for (;;) {
    uint32_t ok;
    asm volatile(
        "{\n.reg .pred p;\n"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    if (ok) return true;
    if (clock64() - t0 > 2000000000ll) {
      if (err) *reinterpret_cast<volatile int*>(err) = 1;
      return false;
    }
  }
}

// Tensor memory: `cols` 32-bit columns (a power of two >= 32) x 128 lanes,
// allocated and freed by one whole warp.
__device__ __forceinline__ void tmem_alloc(uint32_t* slot, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)),
               "r"(cols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_free(uint32_t addr, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(cols) : "memory");
}

__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// generic-proxy shared-memory writes become visible to the tensor core's reads
__device__ __forceinline__ void fence_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// shared-memory operand descriptor: K-major, no swizzle, `lbo` bytes between
// core matrices along K, 128 bytes between row groups
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo) {
  return (uint64_t)((addr >> 4) & 0x3fff) | (uint64_t)((lbo >> 4) & 0x3fff) << 16 |
         (uint64_t)(128 >> 4) << 32 | (uint64_t)1 << 46;
}
// instruction descriptor: M = 128, fp16 A and B, fp32 D
__host__ __device__ constexpr uint32_t idesc_f16(uint32_t n) {
  return (1u << 4) | ((n >> 3) << 17) | ((128u >> 4) << 24);
}
// D[128 x n] (+)= A[128 x 16] B[n x 16]^T
__device__ __forceinline__ void mma_f16(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n.reg .pred p;\n"
      "setp.ne.u32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
      "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
      : "memory");
}
// the barrier completes when every MMA issued so far by this thread has
__device__ __forceinline__ void commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   smem_u32(bar))
               : "memory");
}

// 16 / 8 consecutive columns of the warp's 32 lanes (lane = row)
__device__ __forceinline__ void tmem_ld16(uint32_t addr, float (&v)[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(addr)
      : "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void tmem_ld8(uint32_t addr, float (&v)[8]) {
  uint32_t r[8];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(addr)
               : "memory");
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_zero16(uint32_t addr) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1};" ::"r"(addr),
      "r"(0)
      : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// v = hi + lo with hi = fp16(v), lo = fp16(v - hi): 22 to 23 bits of v while
// lo is a normal number
__device__ __forceinline__ void split8(const float (&v)[8], uint4& hi, uint4& lo) {
  uint32_t h[4], l[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const __half2 a = __floats2half2_rn(v[2 * i], v[2 * i + 1]);
    const float2 b = __half22float2(a);
    const __half2 c = __floats2half2_rn(v[2 * i] - b.x, v[2 * i + 1] - b.y);
    h[i] = *reinterpret_cast<const uint32_t*>(&a);
    l[i] = *reinterpret_cast<const uint32_t*>(&c);
  }
  hi = make_uint4(h[0], h[1], h[2], h[3]);
  lo = make_uint4(l[0], l[1], l[2], l[3]);
}

// Two neighbouring cells added in one 16-byte reduction (16-byte aligned):
// 32 lanes on 8-byte cells of 32 rows ran at 1.5 TB/s, 16 bytes a lane with
// whole 64 / 128-byte segments at 5.5 / 6.3 TB/s.
__device__ __forceinline__ void red_add4(float2* p, float4 v) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w)
               : "memory");
}

// Power-of-two scale 2^-e that brings values of magnitude up to `m` to below 2
// (m = 0: e = 0).  e is held to [-96, 126] so that 2^-e and 2^(e - 28) are
// normal numbers; at 126 values stay below 4.
__device__ __forceinline__ int scale_exp(float m) {
  if (!(m > 0.f)) return 0;
  const int e = (int)(__float_as_uint(m) >> 23) - 127;
  return e < -96 ? -96 : e > 126 ? 126 : e;
}
__device__ __forceinline__ float finite_abs(float v) {  // 0 for infinities and NaN
  const float m = fabsf(v);
  return m <= 3.402823466e38f ? m : 0.f;
}
__device__ __forceinline__ float pow2(int e) { return __uint_as_float((uint32_t)(e + 127) << 23); }

}  // namespace tc
}  // namespace gbn
