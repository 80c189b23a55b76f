// 2D interpolation on the tensor cores (tcgen05), widths w <= 7, over the tiles of
// the tensor-core spreader (gbn_tc_spread.cu):
//
//   D[s, (re/im, transform)] = A[s, cell] B[cell, (re/im, transform)],
//
// A = wx wy over the 16 x 16 cells of a tile, B = the fine cells.  One K step is
// one x row of the tile.  Samples are the rows of D, so a thread ends with the
// values of one sample and neighbouring lanes write neighbouring sorted samples.
// A is MN-major in shared memory (8 samples x 8 cells a core matrix), because the
// weight tables run along the samples.
//
// The gather kernel it replaces (gbn_kernels.cuh, interp_wc) reads every
// footprint through L1, 52 GB for 1024 transforms of 131 072 samples; here a
// tile's cells are read once for up to 128 samples and the weights are formed
// once for 64 transforms.  Bound: the latency of a block (two x rows) of cells
// through conversion, barrier and MMA at two CTAs an SM (tensor memory).
// Stack of stars, 1024 transforms: 4.50 -> 2.24 ms.
//
// Precision as in the spreader: two fp16 parts of every operand, the cross terms
// in accumulators of their own, the mean truncation of the chain given back.
// Fine cells are scaled by the largest of their transform, which the last pass of
// the fused transforms leaves in fmax: an absolute floor of 2^-40 of it.
#include "gbn_internal.cuh"
#include "gbn_tc.cuh"

namespace gbn {

namespace {

using namespace tc;

constexpr int kThreads = 256;
// the epilogue of one value: scale, residual against the data, density
__device__ __forceinline__ void store_value(const InterpArgs& a, int64_t oi, float dj, float2 r) {
  if (a.mode == INTERP_RESID) {
    const float2 ob = a.obs[oi];
    r.x -= ob.x;
    r.y -= ob.y;
    if (a.density) {
      r.x *= dj;
      r.y *= dj;
    }
  }
  a.out[oi] = r;
}

// ---------------------------------------------------------------------------
// CTA = (chunk of <= 128 samples of one tile, group of TG transforms).
// Blocks of 32 cells (two x rows): A by thread = (cell, sample octet), B by
// thread = (transform, x row, y octet); the cells of the next block are on
// their way while this one is formed.
// Tensor memory: [Ah Bh: 2 TG | cross: 2 TG], column = (re/im) * TG + transform.
// ---------------------------------------------------------------------------
constexpr int kChunk2 = kTcChunk2;
constexpr int kTab2 = kChunk2 * 2 + 16;
constexpr int kLboA2 = (kChunk2 / 8) * 128;       // one octet of cells, all samples
constexpr int kAPart2 = 4 * kLboA2;               // hi or lo part of a block
template <int TG>
constexpr int lbo_b2() {
  return 4 * TG * 16 + 32;  // rows hi | lo; + 32: the four cell octets fall into other banks
}
template <int TG>
constexpr size_t smem2() {
  return 2 * (2 * kAPart2 + 4 * (size_t)lbo_b2<TG>()) + 4 * 16 * kTab2;
}

template <int TG>
__global__ void __launch_bounds__(kThreads, 2) interp_tc2d_kernel(InterpArgs a, int* err) {
  constexpr int NM = 2 * TG;
  constexpr uint32_t kCols = 4 * TG < 32 ? 32 : 4 * TG;
  constexpr int LB = lbo_b2<TG>();
  constexpr int kLo = 16 * kTab2;
  constexpr int kBuf = 2 * kAPart2 + 4 * LB;
  extern __shared__ __align__(128) unsigned char sm[];
  unsigned char* const s_wx = sm + 2 * kBuf;       // [hi, lo][16][kTab2]
  unsigned char* const s_wy = s_wx + 2 * kLo;
  __shared__ __align__(8) uint64_t s_bar[2];
  __shared__ uint32_t s_tmem;

  const Geom& g = a.g;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int sub = blockIdx.x;
  const int tile = a.s.sub_bin[sub];
  const int p0 = a.s.sub_start[sub];
  const int cnt = imin(a.s.sub_count[sub], kChunk2);
  const int nty = (g.nkey[1] + g.bs[0] - 1) / g.bs[0];
  const int o0 = (tile / nty) * g.bs[0] - g.koff;
  const int o1 = (tile % nty) * g.bs[0] - g.koff;
  const int c0 = blockIdx.y * TG;
  const int ns = (cnt + 7) >> 3;  // sample octets

  const int si = tid & (kChunk2 - 1);
  const bool yax = tid >= kChunk2;
  float u = 0.f;
  if (si < cnt) u = a.s.u[yax ? 1 : 0][p0 + si];
  for (int i = tid; i < 4 * kLo / 16; i += kThreads)
    reinterpret_cast<uint4*>(s_wx)[i] = make_uint4(0, 0, 0, 0);
  if (tid == 0) {
    bar_init(&s_bar[0]);
    bar_init(&s_bar[1]);
    bar_init_fence();
  }
  if (warp == 0) tmem_alloc(&s_tmem, kCols);

  // the thread's cells: 8 along y of one x row of a block, one transform
  const int bt = tid >> 2, bx = (tid >> 1) & 1, by = tid & 1;
  const bool bon = bt < TG && c0 + bt < a.ntr;
  const float2* const bsrc = a.fine + (int64_t)(c0 + (bon ? bt : 0)) * g.G;
  int by4[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) by4[q] = wrap_once(o1 + 8 * by + 2 * q, g.nf[1]);
  float bf = 0.f;
  if (bon) bf = pow2(14 - scale_exp(__uint_as_float(a.fmax[c0 + bt])));
  float4 f[4];
  auto fetch = [&](int b) {
    const float2* const row = bsrc + (int64_t)wrap_once(o0 + 2 * b + bx, g.nf[0]) * g.nf[1];
#pragma unroll
    for (int q = 0; q < 4; ++q)
      f[q] = bon ? *reinterpret_cast<const float4*>(row + by4[q]) : make_float4(0.f, 0.f, 0.f, 0.f);
  };
  fetch(0);
  __syncthreads();
  if (si < cnt) {
    float wt[7];
    const int i0 = weights_part<7>(u, g, 0, wt) - (yax ? o1 : o0);
    unsigned char* const tab = (yax ? s_wy : s_wx) + 2 * si;
#pragma unroll
    for (int t = 0; t < 7; ++t)
      if (t < g.w) put_split(tab + (i0 + t) * kTab2, kLo, wt[t] * (yax ? kScaleY : kScaleX));
  }
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tm = s_tmem;

  bool ok = true;
  for (int b = 0; b < 8; ++b) {
    unsigned char* const buf = sm + (b & 1) * kBuf;
    if (b >= 2) ok = ok && bar_wait(&s_bar[b & 1], ((b >> 1) - 1) & 1, err);
    if (bt < TG) {
      const float2 s2 = make_float2(bf, bf);
      float re[8], im[8];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float2 x = __fmul2_rn(make_float2(f[q].x, f[q].y), s2);
        const float2 y = __fmul2_rn(make_float2(f[q].z, f[q].w), s2);
        re[2 * q] = x.x;
        im[2 * q] = x.y;
        re[2 * q + 1] = y.x;
        im[2 * q + 1] = y.y;
      }
      if (b < 7) fetch(b + 1);
      unsigned char* const dst = buf + 2 * kAPart2 + (2 * bx + by) * LB + bt * 16;
      uint4 hi, lo;
      split8(re, hi, lo);
      *reinterpret_cast<uint4*>(dst) = hi;
      *reinterpret_cast<uint4*>(dst + NM * 16) = lo;
      split8(im, hi, lo);
      *reinterpret_cast<uint4*>(dst + TG * 16) = hi;
      *reinterpret_cast<uint4*>(dst + (NM + TG) * 16) = lo;
    }
    {
      const unsigned char* const px = s_wx + (2 * b + (lane >> 4)) * kTab2;
      const unsigned char* const py = s_wy + (lane & 15) * kTab2;
      unsigned char* const dst = buf + (lane >> 3) * kLboA2 + (lane & 7) * 16;
      for (int so = warp; so < ns; so += kThreads / 32) {
        uint4 hi, lo;
        mul_split8(*reinterpret_cast<const uint4*>(px + 16 * so), *reinterpret_cast<const uint4*>(px + kLo + 16 * so),
                   *reinterpret_cast<const uint4*>(py + 16 * so), *reinterpret_cast<const uint4*>(py + kLo + 16 * so),
                   hi, lo);
        *reinterpret_cast<uint4*>(dst + so * 128) = hi;
        *reinterpret_cast<uint4*>(dst + kAPart2 + so * 128) = lo;
      }
    }
    fence_async();
    fence_before();
    __syncthreads();
    fence_after();
    if (tid == 0 && ok) {
      const uint32_t ab = smem_u32(buf), bb = ab + 2 * kAPart2;
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const uint64_t db = smem_desc(bb + 2 * k * LB, LB);
        mma_f16(tm, smem_desc(ab + 2 * k * kLboA2, kLboA2), db, idesc_f16(2 * NM) | kMajorA, b + k != 0);
        mma_f16(tm + NM, smem_desc(ab + kAPart2 + 2 * k * kLboA2, kLboA2), db, idesc_f16(NM) | kMajorA, 1);
      }
      commit(&s_bar[b & 1]);
    }
  }
  ok = ok && bar_wait(&s_bar[1], 1, err);  // the eighth block: fourth use of barrier 1
  fence_after();

  // lane = sample; warps 0..3 the first, 4..7 the second half of the transforms
  const int m = 32 * (warp & 3) + lane;
  if (32 * (warp & 3) < cnt && __all_sync(0xffffffffu, ok)) {
    const bool on = m < cnt;
    const int j = on ? a.s.perm[p0 + m] : 0;
    const float dj = on && a.density ? a.density[j] : 1.f;
    const uint32_t tl = tm + ((uint32_t)(32 * (warp & 3)) << 16);
    // mean number of truncated steps, weighted by how much of the sum they see: half of
    // the w x rows of a footprint
    const float lost = 0.5f * (float)g.w * kTrunc;
    const float2 tr = make_float2(lost, lost);
    for (int t0 = (warp >> 2) * (TG / 2); t0 < ((warp >> 2) + 1) * (TG / 2); t0 += 4) {
      if (c0 + t0 >= a.ntr) break;
      float d[2][4], e[2][4];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        tmem_ld4(tl + h * TG + t0, d[h]);
        tmem_ld4(tl + NM + h * TG + t0, e[h]);
      }
      tmem_wait_ld();
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int t = c0 + t0 + q;
        if (t >= a.ntr) break;
        // D is scaled by 2^(29 - e)
        const float sc = pow2(scale_exp(__uint_as_float(a.fmax[t])) - 29) * a.scale;
        const float2 x = make_float2(d[0][q], d[1][q]);
        const float2 v = __fadd2_rn(x, __ffma2_rn(x, tr, make_float2(e[0][q], e[1][q])));
        if (on) store_value(a, (int64_t)t * a.s.M + j, dj, __fmul2_rn(v, make_float2(sc, sc)));
      }
    }
  }
  fence_before();
  __syncthreads();
  fence_after();
  if (warp == 0) tmem_free(tm, kCols);
}

template <int TG>
cudaError_t launch2(const InterpArgs& a, int* err, cudaStream_t st) {
  interp_tc2d_kernel<TG><<<dim3(a.s.nsub, (a.ntr + TG - 1) / TG), kThreads, smem2<TG>(), st>>>(a, err);
  return cudaGetLastError();
}

}  // namespace

cudaError_t tc_interp_prepare() {
  auto set = [](const void* k, size_t b) {
    return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)b);
  };
  cudaError_t e = set((const void*)interp_tc2d_kernel<64>, smem2<64>());
  if (e == cudaSuccess) e = set((const void*)interp_tc2d_kernel<32>, smem2<32>());
  return e;
}

cudaError_t launch_interp_tc(const InterpArgs& a, int* err, cudaStream_t st) {
  if (a.s.nsub == 0) return cudaSuccess;
  return a.ntr > 32 ? launch2<64>(a, err, st) : launch2<32>(a, err, st);
}

}  // namespace gbn
