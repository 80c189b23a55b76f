// Building blocks of the tensor-core kernels: tcgen05 (fp16 operands, fp32
// accumulators in tensor memory), mbarriers, the split of fp32 values into
// two fp16 parts, vector reductions.
//
// Operands lie in shared memory as core matrices of 128 contiguous bytes without
// swizzle: K-major, 8 rows (of M or N) x 8 k values of 16 bytes a row; MN-major,
// 8 k x 8 rows.  The core matrix of row octet r and k octet o sits at
// r * 128 + o * lbo.
#pragma once

#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "gbn_internal.cuh"

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
// instruction descriptor bit: A is MN-major, its core matrices 8 k x 8 rows with
// the rows contiguous
constexpr uint32_t kMajorA = 1u << 15;
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
__device__ __forceinline__ void tmem_ld4(uint32_t addr, float (&v)[4]) {
  uint32_t r[4];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] = __uint_as_float(r[i]);
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
// (m = 0 or infinite: e = 0).  e is held to [-96, 126] so that 2^-e and 2^(e - 28) are
// normal numbers; at 126 values stay below 4.
__device__ __forceinline__ int scale_exp(float m) {
  if (!(m > 0.f) || m > 3.402823466e38f) return 0;
  const int e = (int)(__float_as_uint(m) >> 23) - 127;
  return e < -96 ? -96 : e > 126 ? 126 : e;
}
__device__ __forceinline__ float finite_abs(float v) {  // 0 for infinities and NaN
  const float m = fabsf(v);
  return m <= 3.402823466e38f ? m : 0.f;
}
__device__ __forceinline__ float pow2(int e) { return __uint_as_float((uint32_t)(e + 127) << 23); }

// scales of the split factors: x weights 2^8, y and z weights 2^7, strengths
// 2^(6 - e), fine cells 2^(14 - e) with 2^e the largest of them
constexpr float kScaleX = 256.0f, kScaleY = 128.0f, kScaleC = 64.0f;
// mean relative loss of an accumulator for each step that truncates it, given
// back with the cross terms
constexpr float kTrunc = 6e-8f;
constexpr int kTcRows = 11;   // 3D cross-section rows per axis
constexpr int kRound = 128;   // largest round of samples (3D)

// the w <= 7 kernel weights t0 .. t0 + N - 1 of coordinate u; returns the first cell
template <int N>
__device__ __forceinline__ int weights_part(float u, const Geom& g, int t0, float (&wt)[N]) {
  const int i0 = (int)ceilf(u - g.halfw);
  const float x0 = (float)i0 - u;
#pragma unroll
  for (int t = 0; t < N; ++t)
    wt[t] = t0 + t < g.w ? es_eval(x0 + (float)(t0 + t), g.beta, g.inv_halfw) : 0.f;
  return i0;
}

__device__ __forceinline__ int wrap_once(int i, int n) {
  const int m = i < 0 ? i + n : (i >= n ? i - n : i);
  return (unsigned)m < (unsigned)n ? m : wrap_idx(i, n);
}

// v = hi + lo, stored as halves `lo_off` bytes apart
__device__ __forceinline__ void put_split(unsigned char* p, int lo_off, float v) {
  const __half h = __float2half_rn(v);
  *reinterpret_cast<__half*>(p) = h;
  *reinterpret_cast<__half*>(p + lo_off) = __float2half_rn(v - __half2float(h));
}

// the split product of two split factors, 8 samples: h = xh yh rounded,
// l = (xh yh - h) + xh yl + xl yh, whose first term is exact
__device__ __forceinline__ void mul_split8(const uint4& xh, const uint4& xl, const uint4& yh, const uint4& yl,
                                           uint4& hi, uint4& lo) {
  const uint32_t a[4] = {xh.x, xh.y, xh.z, xh.w}, b[4] = {xl.x, xl.y, xl.z, xl.w};
  const uint32_t c[4] = {yh.x, yh.y, yh.z, yh.w}, d[4] = {yl.x, yl.y, yl.z, yl.w};
  uint32_t h[4], l[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const __half2 p = *reinterpret_cast<const __half2*>(&a[i]), q = *reinterpret_cast<const __half2*>(&b[i]);
    const __half2 r = *reinterpret_cast<const __half2*>(&c[i]), s = *reinterpret_cast<const __half2*>(&d[i]);
    const __half2 u = __hmul2(p, r);
    const __half2 v = __hfma2(q, r, __hfma2(p, s, __hfma2(p, r, __hneg2(u))));
    h[i] = *reinterpret_cast<const uint32_t*>(&u);
    l[i] = *reinterpret_cast<const uint32_t*>(&v);
  }
  hi = make_uint4(h[0], h[1], h[2], h[3]);
  lo = make_uint4(l[0], l[1], l[2], l[3]);
}

// A round of a 3D chunk: up to kRound samples, in z order, cut into groups of one
// z block (first cell + 8) >> 3.  Every group starts at a table column that is
// a multiple of 8; the round ends before column PAD.
struct RoundGroups {
  unsigned start[4];  // bit i: sample i starts a group
  int pads[4];
  int nround, ngrp;   // samples, groups
  short col[kRound];  // table column of a sample
  short gi[kRound + 1], gp[kRound], gz[kRound];  // groups: first sample, column, z block
};

__device__ __forceinline__ int z_block(float u, const Geom& g) { return ((int)ceilf(u - g.halfw) + 8) >> 3; }

// u: the last-axis coordinates of the `left` samples that remain.  Whole CTA
// (at least kRound threads); three barriers, the first before `rg` is read and
// the last after it is complete.
template <int PAD>
__device__ __forceinline__ void round_groups(const float* __restrict__ u, int left, const Geom& g,
                                             RoundGroups& rg) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool have = tid < kRound && tid < left;
  int zb = 0;
  bool start = false;
  if (tid < kRound) {
    if (have) {
      zb = z_block(u[tid], g);
      start = tid == 0 || zb != z_block(u[tid - 1], g);
    }
    const unsigned b = __ballot_sync(0xffffffffu, start);
    if (lane == 0) rg.start[warp] = b;
  }
  __syncthreads();
  // the group start at or before sample i of word w
  auto start_of = [&](int w, unsigned below) {
    while (!below) below = rg.start[--w];
    return 32 * w + 31 - __clz(below);
  };
  int pad = 0, ord = 0;
  if (tid < kRound) {
    // empty columns before a group: the size of the last one up to a multiple of 8
    if (start && tid > 0) pad = (start_of(warp, rg.start[warp] & ((1u << lane) - 1u)) - tid) & 7;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int q = __shfl_up_sync(0xffffffffu, pad, d);
      if (lane >= d) pad += q;
    }
    if (lane == 31) rg.pads[warp] = pad;
  }
  __syncthreads();
  if (tid < kRound) {
    for (int w = 0; w < warp; ++w) {
      pad += rg.pads[w];
      ord += __popc(rg.start[w]);
    }
    const unsigned upto = rg.start[warp] & ((2u << lane) - 1u);
    ord += __popc(upto) - 1;  // the sample's group
    const int c = tid + pad;
    const bool in = have && c < PAD;
    rg.col[tid] = (short)(in ? c : -1);
    if (in && start) {
      rg.gi[ord] = (short)tid;
      rg.gp[ord] = (short)c;
      rg.gz[ord] = (short)zb;
    }
    bool last = in && (tid == kRound - 1 || tid + 1 == left);
    if (in && !last) {  // the last sample before the columns run out
      const bool next = rg.start[(tid + 1) >> 5] >> ((tid + 1) & 31) & 1;
      last = c + 1 + (next ? (start_of(warp, upto) - (tid + 1)) & 7 : 0) >= PAD;
    }
    if (last) {
      rg.nround = tid + 1;
      rg.ngrp = ord + 1;
      rg.gi[ord + 1] = (short)(tid + 1);
    }
  }
  __syncthreads();
}

}  // namespace tc
}  // namespace gbn
