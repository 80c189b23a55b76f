// Spreading on the tensor cores (tcgen05), widths w <= 7.
//
// A tile of neighbouring samples adds rank-one terms to the fine grid, so a
// block of samples is a matrix product.  Both kernels form the operands in
// shared memory, accumulate in tensor memory and add the result to the fine
// grid with 16-byte vector reductions:
//
//   2D  D[cell, (transform, re/im)] += A[cell, s] B[s, (transform, re/im)],
//       A = wx wy over the 16 x 16 cells of a tile of (17 - w)^2 footprint
//       origins, B = the strengths.
//   3D  D[row, (z slot, coil, re/im)] += A[row, s] B[s, (slot, coil, re/im)],
//       A = wx wy over the 11 x 11 rows of a column of (12 - w)^2 origins,
//       B = wz times the strength, the 16 slots a ring along z.
//
// Precision: every operand is split into two fp16 parts (x = hi + lo, 22 to
// 23 bits) and D = Ah Bh + (Ah Bl + Al Bh).  The tensor core truncates when it
// adds to an accumulator (measured: -5.4e-8 of the value for each step of 16
// samples), so the two cross terms, 2^-11 of the first, have accumulators of
// their own, the Ah Bh chain is at most 8 steps long (longer sums continue in
// fp32 on the fine grid), and the mean loss of its steps is given back.  A is
// scaled to 2^15 and B to 2^13 .. 2^15 over the largest strength, which keeps
// the fp16 parts' absolute floor at 2^-32 of the largest value.
#include "gbn_internal.cuh"
#include "gbn_tc.cuh"

namespace gbn {

namespace {

using namespace tc;

constexpr int kThreads = 256;
// ---------------------------------------------------------------------------
// 2D.  CTA = (chunk of <= 128 samples of one tile, group of TG transforms).
// Cell (x, y) of the tile is row 8 x + (y >> 1) of M tile (y & 1), so that a
// thread holds both cells of a 16-byte pair and 8 lanes a 128-byte row.
// Tensor memory: M tile h at columns h * 4 TG: [Ah Bh: 2 TG | cross: 2 TG].
// ---------------------------------------------------------------------------
constexpr int kChunk2 = kTcChunk2;
constexpr int kOct2 = kChunk2 / 8;
constexpr int kTab2 = kChunk2 * 2 + 16;      // row pitch of the weight tables (bytes)
constexpr int kLboA2 = 128 * 16;
constexpr int kABuf2 = 4 * 2 * kLboA2;       // [M tile][hi, lo][2 octets][128 rows][16 B]

template <int TG>
constexpr int lbo_b2() {
  return 4 * TG * 16 + 16;  // + 16: consecutive octets fall into other banks
}
template <int TG>
constexpr size_t smem2() {
  return 2 * kABuf2 + (size_t)kOct2 * lbo_b2<TG>() + 4 * 16 * kTab2 +
         kChunk2 * (sizeof(int) + sizeof(float)) + TG * sizeof(float);
}

template <int TG>
__global__ void __launch_bounds__(kThreads, 2) spread_tc2d_kernel(SpreadArgs a, int* err) {
  constexpr int NM = 2 * TG;                 // columns of one accumulator
  constexpr uint32_t kCols = 8 * TG < 32 ? 32 : 8 * TG;
  constexpr int LB = lbo_b2<TG>();
  constexpr int kLo = 16 * kTab2;            // hi -> lo table
  extern __shared__ __align__(128) unsigned char sm[];
  unsigned char* const s_a = sm;
  unsigned char* const s_b = sm + 2 * kABuf2;
  unsigned char* const s_wx = s_b + kOct2 * LB;                    // [hi, lo][16][kTab2]
  unsigned char* const s_wy = s_wx + 2 * kLo;                      // rows: even y first, then odd
  int* const s_perm = reinterpret_cast<int*>(s_wy + 2 * kLo);
  float* const s_dj = reinterpret_cast<float*>(s_perm + kChunk2);
  float* const s_f = s_dj + kChunk2;                               // result scale per transform
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
  const int nk = (cnt + 15) >> 4;  // K steps

  // thread i < 128: x weights, perm and density of sample i; i + 128: y weights
  const int si = tid & (kChunk2 - 1);
  const bool yax = tid >= kChunk2;
  float u = 0.f;
  if (si < cnt) {
    u = a.s.u[yax ? 1 : 0][p0 + si];
    if (!yax) {
      const int j = a.s.perm[p0 + si];
      s_perm[si] = j;
      s_dj[si] = a.density ? a.scale * a.density[j] : a.scale;
    }
  }
  for (int i = tid; i < 4 * kLo / 16; i += kThreads)
    reinterpret_cast<uint4*>(s_wx)[i] = make_uint4(0, 0, 0, 0);
  if (tid == 0) {
    bar_init(&s_bar[0]);
    bar_init(&s_bar[1]);
    bar_init_fence();
  }
  if (warp == 0) tmem_alloc(&s_tmem, kCols);
  __syncthreads();

  // B: 16 lanes take the 16 sample octets of one transform
  const int o = tid & 15;
  float2 v[(TG + 15) / 16][8];
#pragma unroll
  for (int q = 0; q < (TG + 15) / 16; ++q) {
    const int t = (tid >> 4) + 16 * q;
    const float2* in = a.in + (int64_t)(c0 + t) * a.s.M;
    const bool on = t < TG && c0 + t < a.ntr;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int s = 8 * o + i;
      v[q][i] = make_float2(0.f, 0.f);
      if (on && s < cnt) v[q][i] = in[s_perm[s]];
    }
  }
  if (si < cnt) {  // weights, while the strengths arrive
    float wt[7];
    const int i0 = weights_part<7>(u, g, 0, wt) - (yax ? o1 : o0);
    unsigned char* const tab = (yax ? s_wy : s_wx) + 2 * si;
#pragma unroll
    for (int t = 0; t < 7; ++t) {
      const int r = i0 + t;
      if (t < g.w)
        put_split(tab + (yax ? (r >> 1) + 8 * (r & 1) : r) * kTab2, kLo, wt[t] * (yax ? kScaleY : kScaleX));
    }
  }
#pragma unroll
  for (int q = 0; q < (TG + 15) / 16; ++q) {
    const int t = (tid >> 4) + 16 * q;
    float m = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int s = 8 * o + i;
      const float dj = s < cnt ? s_dj[s] : 0.f;
      if (s < cnt) v[q][i] = make_float2(v[q][i].x * dj, v[q][i].y * dj);
      m = fmaxf(m, fmaxf(finite_abs(v[q][i].x), finite_abs(v[q][i].y)));
    }
#pragma unroll
    for (int d = 1; d < 16; d <<= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, d));
    const int e = scale_exp(m);
    if (t < TG) {
      // B is scaled by 2^(13 - e), the strength's 2^(6 - e) and the z weight's
      // 2^7 of the 3D kernel; in two factors, 13 - e can exceed the exponents
      const float f = pow2(-e), f2 = kScaleC * kScaleY;
      if (o == 0) s_f[t] = pow2(e - 28);
      if (o < 2 * nk) {
        float re[8], im[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          re[i] = v[q][i].x * f * f2;
          im[i] = v[q][i].y * f * f2;
        }
        uint4 hi, lo;
        unsigned char* const dst = s_b + o * LB + 2 * t * 16;
        split8(re, hi, lo);
        *reinterpret_cast<uint4*>(dst) = hi;
        *reinterpret_cast<uint4*>(dst + NM * 16) = lo;
        split8(im, hi, lo);
        *reinterpret_cast<uint4*>(dst + 16) = hi;
        *reinterpret_cast<uint4*>(dst + 16 + NM * 16) = lo;
      }
    }
  }
  fence_before();
  __syncthreads();
  fence_after();

  const uint32_t tm = s_tmem;
  // A, 16 samples at a time: thread = one cell of the tile
  const int h = tid >> 7, m = tid & 127;
  const unsigned char* const px = s_wx + (m >> 3) * kTab2;
  const unsigned char* const py = s_wy + ((m & 7) + 8 * h) * kTab2;
  bool ok = true;
  for (int k = 0; k < nk; ++k) {
    unsigned char* const buf = s_a + (k & 1) * kABuf2;
    if (k >= 2) ok = ok && bar_wait(&s_bar[k & 1], ((k >> 1) - 1) & 1, err);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int off = 32 * k + 16 * q;
      const uint4 xh = *reinterpret_cast<const uint4*>(px + off);
      const uint4 xl = *reinterpret_cast<const uint4*>(px + kLo + off);
      const uint4 yh = *reinterpret_cast<const uint4*>(py + off);
      const uint4 yl = *reinterpret_cast<const uint4*>(py + kLo + off);
      uint4 hi, lo;
      mul_split8(xh, xl, yh, yl, hi, lo);
      unsigned char* const dst = buf + h * 4 * kLboA2 + q * kLboA2 + m * 16;
      *reinterpret_cast<uint4*>(dst) = hi;
      *reinterpret_cast<uint4*>(dst + 2 * kLboA2) = lo;
    }
    fence_async();
    fence_before();
    __syncthreads();
    fence_after();
    if (tid == 0 && ok) {
      const uint32_t bk = smem_u32(s_b) + 2 * k * LB;
      const uint64_t db = smem_desc(bk, LB);
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const uint32_t ak = smem_u32(buf) + q * 4 * kLboA2;
        const uint32_t d = tm + q * 2 * NM;
        mma_f16(d, smem_desc(ak, kLboA2), db, idesc_f16(2 * NM), k != 0);
        mma_f16(d + NM, smem_desc(ak + 2 * kLboA2, kLboA2), db, idesc_f16(NM), 1);
      }
      commit(&s_bar[k & 1]);
    }
  }
  ok = ok && bar_wait(&s_bar[(nk - 1) & 1], ((nk - 1) >> 1) & 1, err);
  fence_after();

  // the tile is added to the fine grids; warps 0..3 the first, 4..7 the second
  // half of the transforms, each on its 32 tensor-memory lanes
  if (__all_sync(0xffffffffu, ok)) {
    const int row = 32 * (warp & 3) + lane;  // M row: cells (row >> 3, 2 (row & 7) + 0, 1)
    const int64_t off = (int64_t)wrap_once(o0 + (row >> 3), g.nf[0]) * g.nf[1] +
                        wrap_once(o1 + 2 * (row & 7), g.nf[1]);
    const uint32_t tl = tm + ((uint32_t)(32 * (warp & 3)) << 16);
    const float2 tr = make_float2(nk * kTrunc, nk * kTrunc);
    for (int t0 = (warp >> 2) * (TG / 2); t0 < ((warp >> 2) + 1) * (TG / 2); t0 += 4) {
      if (c0 + t0 >= a.ntr) break;
      float d[2][8], e[2][8];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        tmem_ld8(tl + 2 * NM * h + 2 * t0, d[h]);
        tmem_ld8(tl + 2 * NM * h + NM + 2 * t0, e[h]);
      }
      tmem_wait_ld();
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (c0 + t0 + q >= a.ntr) break;
        const float f = s_f[t0 + q];
        float2 r[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const float2 x = make_float2(d[h][2 * q], d[h][2 * q + 1]);
          const float2 y = make_float2(e[h][2 * q], e[h][2 * q + 1]);
          r[h] = __fmul2_rn(__fadd2_rn(x, __ffma2_rn(x, tr, y)), make_float2(f, f));
        }
        if (r[0].x != 0.f || r[0].y != 0.f || r[1].x != 0.f || r[1].y != 0.f)
          red_add4(a.fine + (int64_t)(c0 + t0 + q) * g.G + off, make_float4(r[0].x, r[0].y, r[1].x, r[1].y));
      }
    }
  }
  fence_before();
  __syncthreads();
  fence_after();
  if (warp == 0) tmem_free(tm, kCols);
}

// ---------------------------------------------------------------------------
// 3D.  CTA = (chunk of <= 512 samples of one column, in z order, group of 4
// coils).  Cell z sits in slot (z + 8) & 15 of a ring; the samples whose first
// cells share a z block (z + 8) >> 3 of 8 cells reach that block and the next,
// the two halves of the ring.  They are one group: groups are multiplied in
// blocks of up to 32 samples, and before the samples move on to a later z
// block, the halves they leave are added to the fine grid and cleared.  A half
// is also added when its chain of steps gets too long.
//
// Rounds of up to 128 samples have their split weights and strengths tabulated
// at once, every group starting at a multiple of 8 columns.
//
// Tensor memory: columns half * 64 + coil * 16 + slot * 2 + (re, im) of Ah Bh,
// + 128 of the cross terms.
// ---------------------------------------------------------------------------
constexpr int kChunk3 = kTcChunk3;
constexpr int kCoils3 = 4;
constexpr int kRows = kTcRows;
constexpr int kPad = 192;                      // table columns of a round
constexpr int kTabLo = 2 * kPad;               // hi -> lo part of a table row (bytes)
constexpr int kTabP = 4 * kPad + 16;           // row pitch; an odd number of 16-byte units
constexpr int kTabRows = 2 * kRows + 16 + 2 * kCoils3;  // x | y | z by ring slot | strengths
constexpr int kLboA3 = 128 * 16, kLboB3 = 256 * 16;
constexpr int kBuf3 = 4 * (2 * kLboA3 + kLboB3);  // [A hi | A lo | B] of 4 octets: 32 KB
constexpr size_t kSmem3 = 2 * kBuf3 + kTabRows * kTabP;
constexpr int kChain3 = 8;

__global__ void __launch_bounds__(kThreads, 2) spread_tc3d_kernel(SpreadArgs a, int* err) {
  constexpr uint32_t kCols = 256;
  extern __shared__ __align__(128) unsigned char sm[];
  unsigned char* const s_tab = sm + 2 * kBuf3;
  __shared__ __align__(8) uint64_t s_bar[2];
  __shared__ uint32_t s_tmem;
  __shared__ int s_row[128];
  __shared__ unsigned s_max[kCoils3];
  __shared__ RoundGroups rg;

  const Geom& g = a.g;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int sub = blockIdx.x;
  const int col = a.s.sub_bin[sub];
  const int p0 = a.s.sub_start[sub];
  const int cnt = imin(a.s.sub_count[sub], kChunk3);
  const int o0 = (col / g.nb[1]) * g.bs[0] - g.koff;
  const int o1 = (col % g.nb[1]) * g.bs[1] - g.koff;
  const int c0 = blockIdx.y * kCoils3;
  const int nc = imin(kCoils3, a.ntr - c0);
  const int nf2 = g.nf[2];

  if (tid == 0) {
    bar_init(&s_bar[0]);
    bar_init(&s_bar[1]);
    bar_init_fence();
  }
  if (warp == 0) tmem_alloc(&s_tmem, kCols);
  if (tid < kCoils3) s_max[tid] = 0;
  if (tid < 128) {
    const int rx = tid / kRows, ry = tid - rx * kRows;
    s_row[tid] = tid < kRows * kRows
                     ? (wrap_once(o0 + rx, g.nf[0]) * g.nf[1] + wrap_once(o1 + ry, g.nf[1])) * nf2
                     : -1;
  }
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tm = s_tmem;
  const int cp = warp >> 2;  // the warp's coils 2 cp, 2 cp + 1 when the ring is emptied
  const uint32_t tl = tm + ((uint32_t)(32 * (warp & 3)) << 16);

  // largest finite strength of each coil over the chunk
  {
    float m[kCoils3] = {0.f, 0.f, 0.f, 0.f};
    for (int i = tid; i < cnt; i += kThreads) {
      const int j = a.s.perm[p0 + i];
      const float dj = a.density ? a.scale * a.density[j] : a.scale;
#pragma unroll
      for (int c = 0; c < kCoils3; ++c)
        if (c < nc) {
          const float2 x = a.in[(int64_t)(c0 + c) * a.s.M + j];
          m[c] = fmaxf(m[c], fmaxf(finite_abs(x.x * dj), finite_abs(x.y * dj)));
        }
    }
#pragma unroll
    for (int c = 0; c < kCoils3; ++c) {
      const unsigned mm = __reduce_max_sync(0xffffffffu, __float_as_uint(m[c]));
      if (lane == 0) atomicMax(&s_max[c], mm);
    }
  }
#pragma unroll
  for (int q = 0; q < 8; ++q) tmem_zero16(tl + cp * 128 + q * 16);
  tmem_wait_st();

  // adds the ring half of z block `blk` (cells 8 blk - 8 .. 8 blk - 1) to the
  // fine grid and clears it.  Each warp turns its 32 rows through 2 KB of
  // `stage`, so that 4 lanes write one row's 64 bytes.
  auto flush = [&](int blk, int nsteps, unsigned char* stage) {
    unsigned char* const st = stage + warp * 2048;
    const float2 tr = make_float2(nsteps * kTrunc, nsteps * kTrunc);
    const int zc = wrap_once(8 * blk - 8 + 2 * (lane & 3), nf2);
#pragma unroll
    for (int cc = 0; cc < 2; ++cc) {
      const int c = 2 * cp + cc;
      const uint32_t ad = tl + (blk & 1) * 64 + c * 16;
      float v[16], l[16];
      tmem_ld16(ad, v);
      tmem_ld16(ad + 128, l);
      tmem_wait_ld();
      tmem_zero16(ad);
      tmem_zero16(ad + 128);
      if (c >= nc) continue;
      const float f = pow2(scale_exp(__uint_as_float(s_max[c])) - 28);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float2 ff = make_float2(f, f);
        const float2 v0 = make_float2(v[4 * q], v[4 * q + 1]), v1 = make_float2(v[4 * q + 2], v[4 * q + 3]);
        const float2 r0 = __fmul2_rn(
            __fadd2_rn(v0, __ffma2_rn(v0, tr, make_float2(l[4 * q], l[4 * q + 1]))), ff);
        const float2 r1 = __fmul2_rn(
            __fadd2_rn(v1, __ffma2_rn(v1, tr, make_float2(l[4 * q + 2], l[4 * q + 3]))), ff);
        *reinterpret_cast<float4*>(st + lane * 64 + ((q ^ (lane >> 1)) & 3) * 16) =
            make_float4(r0.x, r0.y, r1.x, r1.y);
      }
      __syncwarp();
      float2* const fc = a.fine + (int64_t)(c0 + c) * g.G + zc;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = 8 * i + (lane >> 2);
        const float4 x = *reinterpret_cast<const float4*>(st + r * 64 + (((lane & 3) ^ (r >> 1)) & 3) * 16);
        const int ro = s_row[32 * (warp & 3) + r];
        if (ro >= 0 && (x.x != 0.f || x.y != 0.f || x.z != 0.f || x.w != 0.f)) red_add4(fc + ro, x);
      }
      __syncwarp();
    }
    tmem_wait_st();
  };

  // A: warps 0..3, one octet each; thread = rows lane, lane + 32, ...
  // B: warps 4..7, one octet each; lane = (slot of a half, re/im) of two coils
  const int oc = warp & 3;
  int it = 0, cur = -1;
  int steps[2] = {0, 0};  // steps since the half of z block cur, cur + 1 was cleared
  bool ok = true;

  for (int s0 = 0; s0 < cnt;) {
    // the tables of the last round are consumed (its last block's barrier)
    for (int i = tid; i < kTabRows * kTabP / 16; i += kThreads)
      reinterpret_cast<uint4*>(s_tab)[i] = make_uint4(0, 0, 0, 0);
    round_groups<kPad>(a.s.u[2] + p0 + s0, cnt - s0, g, rg);
    const int nr = rg.nround, ng = rg.ngrp;
    // -- tables: weights of an axis, then strengths of a coil, 32 samples a warp
    for (int q = warp; q < 12 + 4 * kCoils3; q += kThreads / 32) {
      const int i = 32 * (q & 3) + lane;
      if (i >= nr) continue;
      const int pos = p0 + s0 + i;
      unsigned char* const t0 = s_tab + 2 * rg.col[i];
      if (q < 12) {
        const int d = q >> 2;
        float wt[7];
        const int i0 = weights_part<7>(a.s.u[d][pos], g, 0, wt);
        if (d == 2) {
#pragma unroll
          for (int t = 0; t < 7; ++t)
            if (t < g.w) put_split(t0 + (2 * kRows + ((i0 + 8 + t) & 15)) * kTabP, kTabLo, wt[t] * kScaleY);
        } else {
          unsigned char* const p = t0 + (d * kRows + i0 - (d == 0 ? o0 : o1)) * kTabP;
          const float sc = d == 0 ? kScaleX : kScaleY;
#pragma unroll
          for (int t = 0; t < 7; ++t)
            if (t < g.w) put_split(p + t * kTabP, kTabLo, wt[t] * sc);
        }
      } else {
        const int c = (q - 12) >> 2;
        if (c < nc) {
          const int j = a.s.perm[pos];
          const float dj = a.density ? a.scale * a.density[j] : a.scale;
          const float2 x = a.in[(int64_t)(c0 + c) * a.s.M + j];
          const float f = pow2(-scale_exp(__uint_as_float(s_max[c])));
          unsigned char* const p = t0 + (2 * kRows + 16 + 2 * c) * kTabP;
          put_split(p, kTabLo, x.x * dj * f * kScaleC);
          put_split(p + kTabP, kTabLo, x.y * dj * f * kScaleC);
        }
      }
    }
    __syncthreads();

    for (int gr = 0; gr < ng; ++gr) {
      const int ngr = rg.gi[gr + 1] - rg.gi[gr], blk = rg.gz[gr], pc = rg.gp[gr];
      for (int b = 0; b < ngr; b += 32, ++it) {
        const int no = (imin(32, ngr - b) + 7) >> 3;  // octets with samples
        const int nk = (no + 1) >> 1;
        unsigned char* const buf = sm + (it & 1) * kBuf3;
        if (it >= 2) ok = ok && bar_wait(&s_bar[it & 1], ((it >> 1) - 1) & 1, err);
        const unsigned char* const tab = s_tab + 2 * (pc + b + 8 * oc);
        if (oc < no) {
          if (warp < 4) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const int m = lane + 32 * q;
              const int rx = imin(m / kRows, kRows - 1), ry = m % kRows;
              const unsigned char* const px = tab + rx * kTabP;
              const unsigned char* const py = tab + (kRows + ry) * kTabP;
              uint4 hi, lo;
              mul_split8(*reinterpret_cast<const uint4*>(px), *reinterpret_cast<const uint4*>(px + kTabLo),
                         *reinterpret_cast<const uint4*>(py), *reinterpret_cast<const uint4*>(py + kTabLo),
                         hi, lo);
              unsigned char* const dst = buf + oc * kLboA3 + m * 16;
              *reinterpret_cast<uint4*>(dst) = hi;
              *reinterpret_cast<uint4*>(dst + 4 * kLboA3) = lo;
            }
          } else {
            const unsigned char* const tz = tab + (2 * kRows + ((lane >> 1) & 7)) * kTabP;
            const unsigned char* const tc = tab + (2 * kRows + 16 + 2 * (lane >> 4) + (lane & 1)) * kTabP;
            uint4 zh[2], zl[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              zh[h] = *reinterpret_cast<const uint4*>(tz + 8 * h * kTabP);
              zl[h] = *reinterpret_cast<const uint4*>(tz + 8 * h * kTabP + kTabLo);
            }
            unsigned char* const dst = buf + 8 * kLboA3 + oc * kLboB3 + lane * 16;
#pragma unroll
            for (int c = 0; c < 2; ++c) {  // coils 2 c, 2 c + 1
              const uint4 ch = *reinterpret_cast<const uint4*>(tc + 4 * c * kTabP);
              const uint4 cl = *reinterpret_cast<const uint4*>(tc + 4 * c * kTabP + kTabLo);
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                uint4 hi, lo;
                mul_split8(zh[h], zl[h], ch, cl, hi, lo);
                *reinterpret_cast<uint4*>(dst + (h * 64 + c * 32) * 16) = hi;
                *reinterpret_cast<uint4*>(dst + (128 + h * 64 + c * 32) * 16) = lo;
              }
            }
          }
        } else if (oc < 2 * nk) {  // the empty half of the last step
          const uint4 z = make_uint4(0, 0, 0, 0);
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            if (warp < 4) *reinterpret_cast<uint4*>(buf + (oc + 4 * (q & 1)) * kLboA3 + (lane + 32 * (q >> 1)) * 16) = z;
            else *reinterpret_cast<uint4*>(buf + 8 * kLboA3 + oc * kLboB3 + (lane + 32 * q) * 16) = z;
          }
        }
        const bool move = cur >= 0 && blk != cur;
        const bool full = cur >= 0 && !move && steps[0] + nk > kChain3;
        if (move || full) {
          // every MMA so far is done; the other operand buffer is free to stage
          ok = ok && bar_wait(&s_bar[(it - 1) & 1], ((it - 1) >> 1) & 1, err);
          fence_after();
          unsigned char* const stage = sm + ((it - 1) & 1) * kBuf3;
          flush(cur, steps[0], stage);
          steps[0] = 0;
          // the next block's half: left behind, or its chain would get too long
          if (full || blk > cur + 1 || steps[1] + nk > kChain3) {
            flush(cur + 1, steps[1], stage);
            steps[1] = 0;
          }
          if (move) {
            steps[0] = steps[1];
            steps[1] = 0;
          }
        }
        cur = blk;
        steps[0] += nk;
        steps[1] += nk;
        fence_async();
        fence_before();
        __syncthreads();
        fence_after();
        if (tid == 0 && ok) {
          const uint32_t ab = smem_u32(buf), bb = ab + 8 * kLboA3;
          for (int k = 0; k < nk; ++k) {
            const uint64_t db = smem_desc(bb + 2 * k * kLboB3, kLboB3);
            mma_f16(tm, smem_desc(ab + 2 * k * kLboA3, kLboA3), db, idesc_f16(256), 1);
            mma_f16(tm + 128, smem_desc(ab + (4 + 2 * k) * kLboA3, kLboA3), db, idesc_f16(128), 1);
          }
          commit(&s_bar[it & 1]);
        }
      }
    }
    s0 += nr;
  }
  if (it > 0) {
    ok = ok && bar_wait(&s_bar[(it - 1) & 1], ((it - 1) >> 1) & 1, err);
    fence_after();
    if (__all_sync(0xffffffffu, ok)) {
      flush(cur, steps[0], sm);
      flush(cur + 1, steps[1], sm);
    }
  }
  fence_before();
  __syncthreads();
  fence_after();
  if (warp == 0) tmem_free(tm, kCols);
}

template <int TG>
cudaError_t launch2(const SpreadArgs& a, int* err, cudaStream_t st) {
  spread_tc2d_kernel<TG><<<dim3(a.s.nsub, (a.ntr + TG - 1) / TG), kThreads, smem2<TG>(), st>>>(a, err);
  return cudaGetLastError();
}

}  // namespace

cudaError_t tc_spread_prepare() {
  auto set = [](const void* k, size_t b) {
    return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)b);
  };
  cudaError_t e = set((const void*)spread_tc2d_kernel<32>, smem2<32>());
  if (e == cudaSuccess) e = set((const void*)spread_tc2d_kernel<16>, smem2<16>());
  if (e == cudaSuccess) e = set((const void*)spread_tc2d_kernel<8>, smem2<8>());
  if (e == cudaSuccess) e = set((const void*)spread_tc3d_kernel, kSmem3);
  return e;
}

cudaError_t launch_spread_tc(const SpreadArgs& a, int* err, cudaStream_t st) {
  if (a.s.nsub == 0) return cudaSuccess;
  if (a.g.dim == 3) {
    spread_tc3d_kernel<<<dim3(a.s.nsub, (a.ntr + kCoils3 - 1) / kCoils3), kThreads, kSmem3, st>>>(a, err);
    return cudaGetLastError();
  }
  // the widest group that the transforms fill: A is formed once per group
  if (a.ntr > 16) return launch2<32>(a, err, st);
  return a.ntr > 8 ? launch2<16>(a, err, st) : launch2<8>(a, err, st);
}

}  // namespace gbn
