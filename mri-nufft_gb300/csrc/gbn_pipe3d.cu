// The pipe density iteration on real grids, 3D.
//
// w <- w / |interp(spread(w))| starts from real weights and the kernel is real, so
// the grid and every later w are real: half the cells' bytes, multiply-adds and
// shared-memory reads of the complex kernels.
#include "gbn_kernels.cuh"

namespace gbn {

namespace {

// Spread of one real strength a sample: the quadrant-streaming kernel (see
// spread_quad3d_kernel) for real cells.  One transform pays its per-sample work
// (fetch, row test, weights) for few multiply-adds, so the kernel is bound by
// issue slots.  A thread owns two neighbouring rows along y, 8 cells of the z
// window each: a quadrant's (3 + W)^2 rows are at most 50 threads, two warps that
// each sample costs about 25 instructions (the complex kernel: 3.25 warps of about
// 40).  Row weights are staged by row, zero outside the footprint, the strength in
// the x ones; the window's z cells pair up for the two-wide multiply-adds.
// 2.1 M samples on 128^3 cells: 603 -> 326 us; rounds of 128 samples at 12 CTAs per
// SM 392, of 64 at 16 CTAs 337, at 20 326.
constexpr int kRealThreads = 64;
constexpr int kRealRound = 64;  // samples staged at a time
constexpr int kRowPitch = 12;    // >= 3 + 7 rows, 16-byte rows

template <int W>
__global__ void __launch_bounds__(kRealThreads, 20) spread_real3d_kernel(SpreadArgs a) {
  constexpr int kRows = 3 + W, kPairs = (kRows + 1) / 2;
  static_assert(W <= 7 && kRows * kPairs <= kRealThreads && kRows < kRowPitch, "");
  __shared__ __align__(16) float s_w0[kRealRound * kRowPitch];
  __shared__ __align__(16) float s_w1[kRealRound * kRowPitch];
  __shared__ __align__(16) float s_w2[kRealRound * 8];  // slot order
  // window anchor; x rows (bits 0-15) and y row pairs (from bit 16) of the footprint
  __shared__ int2 s_hd[kRealRound];
  __shared__ short s_list[kStreamBatch];  // chunk indices, z order
  __shared__ int s_wsum[kRealThreads / 32];

  const Geom& g = a.g;
  const float* const in = reinterpret_cast<const float*>(a.in);
  const int sub = blockIdx.x >> 2;
  const int col = a.s.sub_bin[sub];
  const int p0 = a.s.sub_start[sub];
  const int cnt = imin(a.s.sub_count[sub], kStreamBatch);
  const int qx = (blockIdx.x >> 1) & 1, qy = blockIdx.x & 1;
  const int b0 = (col / g.nb[1]) * g.bs[0] - g.koff;  // column origin
  const int b1 = (col % g.nb[1]) * g.bs[1] - g.koff;
  const int o0 = b0 + 4 * qx, o1 = b1 + 4 * qy;       // quadrant origin
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  // the chunk's samples whose footprint starts in this quadrant, in order: warp w
  // looks through half w of the chunk, all its coordinates loaded at once
  constexpr int kHalf = kStreamBatch / 2;
  unsigned mine = 0;  // bit q: sample half + 32 q + lane
  {
    float u0[kHalf / 32], u1[kHalf / 32];
#pragma unroll
    for (int q = 0; q < kHalf / 32; ++q) {
      const int t = warp * kHalf + 32 * q + lane;
      u0[q] = t < cnt ? a.s.u[0][p0 + t] : 0.f;
      u1[q] = t < cnt ? a.s.u[1][p0 + t] : 0.f;
    }
#pragma unroll
    for (int q = 0; q < kHalf / 32; ++q) {
      const int a0 = (int)ceilf(u0[q] - g.halfw) - b0;  // 0 .. 7
      const int a1 = (int)ceilf(u1[q] - g.halfw) - b1;
      const bool in_q = warp * kHalf + 32 * q + lane < cnt && (a0 >= 4) == (qx == 1) && (a1 >= 4) == (qy == 1);
      mine |= in_q ? 1u << q : 0u;
    }
  }
  int count = 0;
#pragma unroll
  for (int q = 0; q < kHalf / 32; ++q) count += __popc(__ballot_sync(0xffffffffu, (mine >> q) & 1u));
  if (lane == 0) s_wsum[warp] = count;
  __syncthreads();
  const int n_own = s_wsum[0] + s_wsum[1];
  int before = warp ? s_wsum[0] : 0;
#pragma unroll
  for (int q = 0; q < kHalf / 32; ++q) {
    const bool m = (mine >> q) & 1u;
    const unsigned bal = __ballot_sync(0xffffffffu, m);
    if (m) s_list[before + __popc(bal & ((1u << lane) - 1u))] = (short)(warp * kHalf + 32 * q + lane);
    before += __popc(bal);
  }
  __syncthreads();
  if (n_own == 0) return;

  const bool own = (int)threadIdx.x < kRows * kPairs;
  const int i0 = own ? threadIdx.x / kPairs : 0, jp = own ? threadIdx.x - i0 * kPairs : 0;
  const unsigned mybits = (1u << i0) | (0x10000u << jp);
  const int nf2 = g.nf[2];
  const int x = wrap_idx(o0 + i0, g.nf[0]) * g.nf[1];
  float* const row0 = reinterpret_cast<float*>(a.fine) + (x + wrap_idx(o1 + 2 * jp, g.nf[1])) * (int64_t)nf2;
  float* const row1 = reinterpret_cast<float*>(a.fine) + (x + wrap_idx(o1 + 2 * jp + 1, g.nf[1])) * (int64_t)nf2;

  float2 acc[2][4];  // [row][slots 2 k, 2 k + 1]
#pragma unroll
  for (int k = 0; k < 4; ++k) acc[0][k] = acc[1][k] = make_float2(0.f, 0.f);
  int zb = 0;  // window: cells zb .. zb + 7, cell z in slot z & 7
  auto flush = [&](unsigned mask) {
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      if (mask & (1u << k)) {
        const int z = wrap_near(zb + ((k - zb) & 7), nf2);
        float& v0 = (k & 1) ? acc[0][k >> 1].y : acc[0][k >> 1].x;
        float& v1 = (k & 1) ? acc[1][k >> 1].y : acc[1][k >> 1].x;
        if (v0 != 0.f) atomicAdd(row0 + z, v0);
        if (v1 != 0.f) atomicAdd(row1 + z, v1);
        v0 = v1 = 0.f;
      }
    }
  };
  for (int r0 = 0; r0 < n_own; r0 += kRealRound) {
    const int nr = imin(kRealRound, n_own - r0);
    if (r0) __syncthreads();  // the previous round is consumed
    for (int t = threadIdx.x; t < nr; t += kRealThreads) {
      const int pos = p0 + s_list[r0 + t];
      const int j = a.s.perm[pos];
      const float c = a.scale * in[j];
      float4* const z0 = reinterpret_cast<float4*>(s_w0 + t * kRowPitch);
      float4* const z1 = reinterpret_cast<float4*>(s_w1 + t * kRowPitch);
#pragma unroll
      for (int k = 0; k < kRowPitch / 4; ++k) z0[k] = z1[k] = make_float4(0.f, 0.f, 0.f, 0.f);
      float wt[W];
      const int a0 = weights_rt<W>(a.s.u[0][pos], g, wt) - o0;  // 0 .. 3
#pragma unroll
      for (int k = 0; k < W; ++k) s_w0[t * kRowPitch + a0 + k] = c * wt[k];
      const int a1 = weights_rt<W>(a.s.u[1][pos], g, wt) - o1;
#pragma unroll
      for (int k = 0; k < W; ++k) s_w1[t * kRowPitch + a1 + k] = wt[k];
      const int zs = weights_rt<W>(a.s.u[2][pos], g, wt);
#pragma unroll
      for (int k = 0; k < 8; ++k) s_w2[t * 8 + ((zs + k) & 7)] = k < W ? wt[k] : 0.f;
      const int pa = a1 >> 1, pb = (a1 + W - 1) >> 1;
      s_hd[t] = make_int2(zs, (((1 << W) - 1) << a0) | (((1 << (pb - pa + 1)) - 1) << (16 + pa)));
    }
    __syncthreads();
    if (!own) continue;
    if (r0 == 0) zb = s_hd[0].x;
#pragma unroll 1
    for (int s = 0; s < nr; ++s) {
      const int2 hd = s_hd[s];
      if (hd.x != zb) {  // the same for every thread: flush the cells that leave the window
        const int steps = imin(hd.x - zb, 8);
        const unsigned m = (1u << steps) - 1u, r = (unsigned)zb & 7u;
        flush(((m << r) | (m >> (8u - r))) & 0xffu);
        zb = hd.x;
      }
      if (((unsigned)hd.y & mybits) == mybits) {
        const float w0 = s_w0[s * kRowPitch + i0];
        const float2 w1 = *reinterpret_cast<const float2*>(s_w1 + s * kRowPitch + 2 * jp);
        const float4* w4 = reinterpret_cast<const float4*>(s_w2 + s * 8);
        const float4 wa = w4[0], wb = w4[1];
        const float2 wz[4] = {make_float2(wa.x, wa.y), make_float2(wa.z, wa.w), make_float2(wb.x, wb.y),
                              make_float2(wb.z, wb.w)};
        const float k0 = w0 * w1.x, k1 = w0 * w1.y;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          acc[0][k] = __ffma2_rn(make_float2(k0, k0), wz[k], acc[0][k]);
          acc[1][k] = __ffma2_rn(make_float2(k1, k1), wz[k], acc[1][k]);
        }
      }
    }
  }
  if (own) flush(0xffu);
}

// The tile kernel on real cells: 338 -> 230 us on the same samples (8 CTAs per SM;
// 234 at 7); two thirds of its instructions are weights, lane order and tile loads.
template <int W>
__global__ void __launch_bounds__(kInterpThreads, 8) interp_real3d_kernel(InterpArgs a) {
  interp_body<3, W, 1, float>(a, blockIdx.x);
}

template <int W>
cudaError_t spread_w(const SpreadArgs& a, cudaStream_t st) {
  spread_real3d_kernel<W><<<(unsigned)(4 * (int64_t)a.s.nsub), kRealThreads, 0, st>>>(a);
  return cudaGetLastError();
}
template <int W>
cudaError_t interp_w(const InterpArgs& a, cudaStream_t st) {
  const size_t smem = (size_t)a.g.tile * sizeof(float);
  cudaError_t e = cudaFuncSetAttribute(interp_real3d_kernel<W>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)smem);
  if (e != cudaSuccess) return e;
  interp_real3d_kernel<W><<<a.s.nsub, kInterpThreads, smem, st>>>(a);
  return cudaGetLastError();
}
}  // namespace

cudaError_t launch_spread_real3d(const SpreadArgs& a, cudaStream_t st) {
  if (a.s.nsub == 0) return cudaSuccess;
  switch (a.g.w) {
    case 7: return spread_w<7>(a, st);
    case 6: return spread_w<6>(a, st);
    case 5: return spread_w<5>(a, st);
    case 4: return spread_w<4>(a, st);
  }
  return cudaErrorInvalidValue;
}

cudaError_t launch_interp_real3d(const InterpArgs& a, cudaStream_t st) {
  if (a.s.nsub == 0) return cudaSuccess;
  switch (a.g.w) {
    case 7: return interp_w<7>(a, st);
    case 6: return interp_w<6>(a, st);
    case 5: return interp_w<5>(a, st);
    case 4: return interp_w<4>(a, st);
  }
  return cudaErrorInvalidValue;
}

}  // namespace gbn
