// Stacked NUFFT z-axis passes (stack-of-stars / stack-of-spirals).
//
// mri-nufft's stacked operator (src/mrinufft/operators/stacked.py:178-330)
// applies, per coil, a centred orthonormal DFT along the last image axis
// (fftshift(fft(ifftshift(x), norm="ortho")) / sqrt(2)), keeps the z_index
// planes, and runs a 2D NUFFT on every kept plane of every coil; the adjoint
// scatters the planes back, inverts the DFT and combines the coils.  Here
// the passes around cuFFT are fused kernels:
//   forward: pad    P[c][x][y][(z - h) mod Nz] = (s_c x)[x][y][z]   (h = Nz/2)
//            cuFFT along z (C Nx Ny transforms of Nz contiguous cells)
//            gather out[c NZ + k][x][y] = P[c][x][y][(zi_k - h) mod Nz] / sqrt(2 Nz)
//   adjoint: scatter (zero P, then the kept planes / sqrt(2 Nz)),
//            inverse cuFFT along z,
//            crop  img[x][y][z] = sum_c conj(s_c) P[c][x][y][(z - h) mod Nz]
//            (calibless: one image per coil).
//
// Stacks of up to about 128 planes do each direction in one kernel instead: 32
// (x, y) columns of a CTA go through shared memory, the z transform is a sum over
// Nz / R terms per plane after one radix-R step (R = 4, 2 or 1, the largest that
// divides Nz), and the work stack is never written: 1.1 GB a direction instead of
// 3.2 GB for 256 x 256 x 64 and 16 coils, op + adj around the 2D transforms 3.2 ->
// 1.0 ms (floor at the copy bandwidth 0.33; the forward sum is FP32-bound).  Their work
// grows with planes squared, so long odd axes and small stacks keep the three passes
// (fwd_in_one, adj_in_one).
#include <cufft.h>

#include <cmath>
#include <map>
#include <string>
#include <vector>

#include "gbnufft.h"
#include "gbn_internal.cuh"

namespace gbn {
namespace {

struct StackGeom {
  int nx, ny, nz;  // image shape (z is the stacked, last axis)
  int nzi;         // kept planes
  int64_t nxy;     // nx * ny
  int64_t nimg;    // nx * ny * nz
};

__device__ __forceinline__ float2 cmul_(float2 a, float2 b) {
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ float2 cmulc_(float2 a, float2 b) {  // conj(a) * b
  return make_float2(a.x * b.x + a.y * b.y, a.x * b.y - a.y * b.x);
}

// one thread per (c, x, y, z) cell of the padded stack
__global__ void stack_pad_kernel(StackGeom g, const float2* __restrict__ img,
                                 const float2* __restrict__ smaps, float2* __restrict__ P, int C) {
  const int64_t total = (int64_t)C * g.nimg;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t c = i / g.nimg;
    const int64_t r = i - c * g.nimg;  // (x, y, z) of the image, z fastest
    const int z = (int)(r % g.nz);
    const int64_t col = r / g.nz;
    float2 v;
    if (smaps) v = cmul_(img[r], smaps[i]);
    else v = img[i];
    int zz = z - g.nz / 2;
    if (zz < 0) zz += g.nz;
    P[(c * g.nxy + col) * g.nz + zz] = v;
  }
}

// one thread per (c, k, x, y) output cell
__global__ void stack_gather_kernel(StackGeom g, const float2* __restrict__ P,
                                    const int* __restrict__ zpos, float2* __restrict__ out, int C,
                                    float scale) {
  const int64_t total = (int64_t)C * g.nzi * g.nxy;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t plane = i / g.nxy;  // c * nzi + k
    const int64_t col = i - plane * g.nxy;
    const int64_t c = plane / g.nzi;
    const int k = (int)(plane - c * g.nzi);
    const float2 v = P[(c * g.nxy + col) * g.nz + zpos[k]];
    out[i] = make_float2(v.x * scale, v.y * scale);
  }
}

// adjoint of the gather: P (zeroed by the caller) at the kept planes
__global__ void stack_scatter_kernel(StackGeom g, const float2* __restrict__ in,
                                     const int* __restrict__ zpos, float2* __restrict__ P, int C,
                                     float scale) {
  const int64_t total = (int64_t)C * g.nzi * g.nxy;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t plane = i / g.nxy;
    const int64_t col = i - plane * g.nxy;
    const int64_t c = plane / g.nzi;
    const int k = (int)(plane - c * g.nzi);
    const float2 v = in[i];
    P[(c * g.nxy + col) * g.nz + zpos[k]] = make_float2(v.x * scale, v.y * scale);
  }
}

// adjoint of the pad: coil combine (SENSE) or per-coil images
__global__ void stack_crop_kernel(StackGeom g, const float2* __restrict__ P,
                                  const float2* __restrict__ smaps, float2* __restrict__ img, int C,
                                  int accumulate) {
  const int64_t total = smaps ? g.nimg : (int64_t)C * g.nimg;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t c0 = smaps ? 0 : i / g.nimg;
    const int64_t r = i - c0 * g.nimg;
    const int z = (int)(r % g.nz);
    const int64_t col = r / g.nz;
    int zz = z - g.nz / 2;
    if (zz < 0) zz += g.nz;
    float2 acc;
    if (smaps) {
      acc = make_float2(0.f, 0.f);
      for (int c = 0; c < C; ++c) {
        const float2 p = cmulc_(smaps[(int64_t)c * g.nimg + r], P[((int64_t)c * g.nxy + col) * g.nz + zz]);
        acc.x += p.x;
        acc.y += p.y;
      }
    } else {
      acc = P[(c0 * g.nxy + col) * g.nz + zz];
    }
    if (accumulate) {
      const float2 o = img[i];
      acc.x += o.x;
      acc.y += o.y;
    }
    img[i] = acc;
  }
}

// ---------------------------------------------------------------------------
// One-kernel z transforms.  With n4 = Nz / R and z = z' + p n4 (positions of the
// shifted axis), plane f = zpos is
//   X[f] = sum_{z' < n4} W^(f z') t_{f mod R}[z'],  t_r[z'] = sum_p v[z' + p n4] i_R^(-r p),
// i_R = exp(2 pi i / R).  `order` lists the kept planes by f mod R in groups of 8
// of one residue (-1: padding), W[z'][j] = exp(-2 pi i f_j z' / Nz) (0: padding).
// Lane = column throughout.
// ---------------------------------------------------------------------------
struct StackDft {
  const float2* W;     // n4 x npad
  const int* order;    // npad
  int n4, npad;
};
constexpr int kDftCols = 32;
constexpr int kDftThreads = 256;
constexpr int kDftWarps = kDftThreads / 32;

__device__ __forceinline__ float2 rot_m(float2 v, int q) {  // v * (-i)^q
  switch (q & 3) {
    case 0: return v;
    case 1: return make_float2(v.y, -v.x);
    case 2: return make_float2(-v.x, -v.y);
    default: return make_float2(-v.y, v.x);
  }
}

// grid: columns / 32, coils
template <int R>
__global__ void __launch_bounds__(kDftThreads)
stack_fwd_dft_kernel(StackGeom g, StackDft d, const float2* __restrict__ img,
                     const float2* __restrict__ smaps, float2* __restrict__ out, float scale) {
  extern __shared__ __align__(16) float2 s_dft[];
  float2* const s_w = s_dft;                       // [n4][npad]
  float2* const s_v = s_w + d.n4 * d.npad;         // [nz][33]
  constexpr int P = kDftCols + 1;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t col0 = (int64_t)blockIdx.x * kDftCols;
  const int ncol = g.nxy - col0 < kDftCols ? (int)(g.nxy - col0) : kDftCols;
  const int c = blockIdx.y;
  for (int i = threadIdx.x; i < d.n4 * d.npad; i += kDftThreads) s_w[i] = d.W[i];
  const float2* const src = (smaps ? img : img + (int64_t)c * g.nimg) + col0 * g.nz;
  const float2* const map = smaps ? smaps + (int64_t)c * g.nimg + col0 * g.nz : nullptr;
  for (int i = threadIdx.x; i < kDftCols * g.nz; i += kDftThreads) {
    const int cl = i / g.nz, z = i - cl * g.nz;
    float2 v = make_float2(0.f, 0.f);
    if (cl < ncol) {
      v = src[i];
      if (map) v = cmul_(v, map[i]);
    }
    int zz = z - g.nz / 2;
    if (zz < 0) zz += g.nz;
    s_v[zz * P + cl] = v;
  }
  __syncthreads();
  if (R > 1) {
    for (int z = warp; z < d.n4; z += kDftWarps) {
      float2 v[R], t[R];
#pragma unroll
      for (int p = 0; p < R; ++p) v[p] = s_v[(z + p * d.n4) * P + lane];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        t[r] = v[0];
#pragma unroll
        for (int p = 1; p < R; ++p) {
          const float2 w = rot_m(v[p], (4 / R) * r * p);
          t[r].x += w.x;
          t[r].y += w.y;
        }
      }
#pragma unroll
      for (int r = 0; r < R; ++r) s_v[(z + r * d.n4) * P + lane] = t[r];
    }
    __syncthreads();
  }
  for (int j0 = 8 * warp; j0 < d.npad; j0 += 8 * kDftWarps) {
    const int r = R == 1 ? 0 : d.order[j0] & (R - 1);  // the group's residue (low bits of order)
    float2 acc[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] = make_float2(0.f, 0.f);
    const float2* const t = s_v + r * d.n4 * P + lane;
    for (int z = 0; z < d.n4; ++z) {
      const float2 v = t[z * P];
      const float2 iv = make_float2(-v.y, v.x);
      const float4* const w4 = reinterpret_cast<const float4*>(s_w + z * d.npad + j0);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float4 w = w4[q];
        acc[2 * q] = __ffma2_rn(make_float2(w.x, w.x), v, acc[2 * q]);
        acc[2 * q] = __ffma2_rn(make_float2(w.y, w.y), iv, acc[2 * q]);
        acc[2 * q + 1] = __ffma2_rn(make_float2(w.z, w.z), v, acc[2 * q + 1]);
        acc[2 * q + 1] = __ffma2_rn(make_float2(w.w, w.w), iv, acc[2 * q + 1]);
      }
    }
    if (lane < ncol) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int k = d.order[j0 + j] >> 2;
        if (k >= 0)
          out[((int64_t)c * g.nzi + k) * g.nxy + col0 + lane] = make_float2(acc[j].x * scale, acc[j].y * scale);
      }
    }
  }
}

// grid: columns / 32 (SENSE: every coil in turn, summed), x coils without maps
template <int R>
__global__ void __launch_bounds__(kDftThreads)
stack_adj_dft_kernel(StackGeom g, StackDft d, const float2* __restrict__ in,
                     const float2* __restrict__ smaps, float2* __restrict__ img, int C, int accumulate,
                     float scale) {
  constexpr int ZP = 16 / R;  // z' of a warp: n4 <= 8 ZP
  extern __shared__ __align__(16) float2 s_dft[];
  float2* const s_w = s_dft;                            // [n4][npad]
  float2* const s_in = s_w + d.n4 * d.npad;             // [npad][32]
  float2* const s_m = s_in + d.npad * kDftCols;         // [32][nz + 1], maps, then the result
  const int mp = g.nz + 1 + (g.nz & 1);                 // odd pitch
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t col0 = (int64_t)blockIdx.x * kDftCols;
  const int ncol = g.nxy - col0 < kDftCols ? (int)(g.nxy - col0) : kDftCols;
  const int cb = smaps ? 0 : blockIdx.y, ce = smaps ? C : cb + 1;
  for (int i = threadIdx.x; i < d.n4 * d.npad; i += kDftThreads) s_w[i] = d.W[i];
  float2 acc[ZP][R];
#pragma unroll
  for (int q = 0; q < ZP; ++q)
#pragma unroll
    for (int p = 0; p < R; ++p) acc[q][p] = make_float2(0.f, 0.f);
  for (int c = cb; c < ce; ++c) {
    __syncthreads();  // the last coil's planes and maps are consumed
    for (int j = warp; j < d.npad; j += kDftWarps) {
      const int k = d.order[j] >> 2;
      float2 v = make_float2(0.f, 0.f);
      if (k >= 0 && lane < ncol) v = in[((int64_t)c * g.nzi + k) * g.nxy + col0 + lane];
      s_in[j * kDftCols + lane] = v;
    }
    if (smaps) {
      const float2* const map = smaps + (int64_t)c * g.nimg + col0 * g.nz;
      for (int i = threadIdx.x; i < ncol * g.nz; i += kDftThreads) {
        const int cl = i / g.nz;
        s_m[cl * mp + (i - cl * g.nz)] = map[i];
      }
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < ZP; ++q) {
      const int z = warp + kDftWarps * q;
      if (z >= d.n4) break;
      float2 S[R];
#pragma unroll
      for (int r = 0; r < R; ++r) S[r] = make_float2(0.f, 0.f);
      for (int j0 = 0; j0 < d.npad; j0 += 8) {
        float2 t = make_float2(0.f, 0.f);
        const float4* const w4 = reinterpret_cast<const float4*>(s_w + z * d.npad + j0);
#pragma unroll
        for (int e = 0; e < 4; ++e) {  // conj(W) v
          const float4 w = w4[e];
          const float2 a = s_in[(j0 + 2 * e) * kDftCols + lane], b = s_in[(j0 + 2 * e + 1) * kDftCols + lane];
          t = __ffma2_rn(make_float2(w.x, w.x), a, t);
          t = __ffma2_rn(make_float2(w.y, w.y), make_float2(a.y, -a.x), t);
          t = __ffma2_rn(make_float2(w.z, w.z), b, t);
          t = __ffma2_rn(make_float2(w.w, w.w), make_float2(b.y, -b.x), t);
        }
        const int r = R == 1 ? 0 : d.order[j0] & (R - 1);
#pragma unroll
        for (int e = 0; e < R; ++e)
          if (r == e) {
            S[e].x += t.x;
            S[e].y += t.y;
          }
      }
#pragma unroll
      for (int p = 0; p < R; ++p) {
        float2 v = S[0];
#pragma unroll
        for (int r = 1; r < R; ++r) {
          const float2 w = rot_m(S[r], 4 - (4 / R) * r * p % 4);  // S_r i_R^(r p)
          v.x += w.x;
          v.y += w.y;
        }
        if (smaps) {
          int zi = z + p * d.n4 + g.nz / 2;
          if (zi >= g.nz) zi -= g.nz;
          if (lane < ncol) v = cmulc_(s_m[lane * mp + zi], v);
        }
        acc[q][p].x += v.x;
        acc[q][p].y += v.y;
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < ZP; ++q) {
    const int z = warp + kDftWarps * q;
    if (z >= d.n4) break;
#pragma unroll
    for (int p = 0; p < R; ++p) {
      int zi = z + p * d.n4 + g.nz / 2;
      if (zi >= g.nz) zi -= g.nz;
      s_m[lane * mp + zi] = make_float2(acc[q][p].x * scale, acc[q][p].y * scale);
    }
  }
  __syncthreads();
  float2* const dst = img + (int64_t)cb * g.nimg + col0 * g.nz;
  for (int i = threadIdx.x; i < ncol * g.nz; i += kDftThreads) {
    const int cl = i / g.nz;
    float2 v = s_m[cl * mp + (i - cl * g.nz)];
    if (accumulate) {
      v.x += dst[i].x;
      v.y += dst[i].y;
    }
    dst[i] = v;
  }
}

template <int R>
cudaError_t dft_fwd(const StackGeom& g, const StackDft& d, const float2* img, const float2* smaps, float2* out,
                    int C, float scale, size_t smem, cudaStream_t st) {
  stack_fwd_dft_kernel<R><<<dim3((unsigned)((g.nxy + kDftCols - 1) / kDftCols), C), kDftThreads, smem, st>>>(
      g, d, img, smaps, out, scale);
  return cudaGetLastError();
}
template <int R>
cudaError_t dft_adj(const StackGeom& g, const StackDft& d, const float2* in, const float2* smaps, float2* img,
                    int C, int accumulate, float scale, size_t smem, cudaStream_t st) {
  stack_adj_dft_kernel<R>
      <<<dim3((unsigned)((g.nxy + kDftCols - 1) / kDftCols), smaps ? 1 : C), kDftThreads, smem, st>>>(
          g, d, in, smaps, img, C, accumulate, scale);
  return cudaGetLastError();
}

unsigned blocks_for(int64_t n) {
  int64_t b = (n + 255) / 256;
  if (b < 1) b = 1;
  if (b > 152 * 64) b = 152 * 64;
  return (unsigned)b;
}

}  // namespace
}  // namespace gbn

using namespace gbn;

struct gbn_stack_s {
  StackGeom g{};
  int device = 0;
  int* zpos = nullptr;     // kept planes as positions in the shifted z axis
  float2* P = nullptr;     // C x nx x ny x nz work stack
  int64_t pcap = 0;        // cells of P
  std::map<int, cufftHandle> ffts;
  int radix = 0;           // one-kernel z transforms: R (0: pad, cuFFT and gather)
  StackDft dft{};
  float2* W = nullptr;
  int* order = nullptr;
  size_t smem_fwd = 0, smem_adj = 0;
  ~gbn_stack_s() {
    int prev = -1;
    cudaGetDevice(&prev);
    if (prev != device) cudaSetDevice(device);
    for (auto& kv : ffts) cufftDestroy(kv.second);
    if (zpos) cudaFree(zpos);
    if (P) cudaFree(P);
    if (W) cudaFree(W);
    if (order) cudaFree(order);
    if (prev >= 0 && prev != device) cudaSetDevice(prev);
  }
};

namespace {

int stack_fail(int code, const std::string& msg) {
  set_last_error(msg.c_str());
  return code;
}

int ck_cuda(cudaError_t e, const char* what) {
  if (e == cudaSuccess) return GBN_OK;
  cudaGetLastError();
  return stack_fail(e == cudaErrorMemoryAllocation ? GBN_ERR_NOMEM : GBN_ERR_CUDA,
                    std::string(what) + ": " + cudaGetErrorString(e));
}

struct DevSwitch {
  int prev = -1;
  explicit DevSwitch(int dev) {
    cudaGetDevice(&prev);
    if (prev != dev) cudaSetDevice(dev);
  }
  ~DevSwitch() {
    int cur = -1;
    cudaGetDevice(&cur);
    if (prev >= 0 && cur != prev) cudaSetDevice(prev);
  }
};

// work stack and z-FFT plan for C coils
int stack_prepare(gbn_stack s, int C, cufftHandle* plan) {
  const int64_t need = (int64_t)C * s->g.nimg;
  if (need > s->pcap) {
    if (s->P) cudaFree(s->P);
    s->P = nullptr;
    s->pcap = 0;
    int rc = ck_cuda(cudaMalloc(&s->P, sizeof(float2) * need), "stack work array");
    if (rc) return rc;
    s->pcap = need;
  }
  auto it = s->ffts.find(C);
  if (it == s->ffts.end()) {
    cufftHandle h;
    int n[1] = {s->g.nz};
    const int64_t batch = (int64_t)C * s->g.nxy;
    if (batch > 0x7fffffff) return stack_fail(GBN_ERR_ARG, "stack too large for one z-FFT plan");
    cufftResult r = cufftPlanMany(&h, 1, n, nullptr, 1, s->g.nz, nullptr, 1, s->g.nz, CUFFT_C2C,
                                  (int)batch);
    if (r != CUFFT_SUCCESS)
      return stack_fail(r == CUFFT_ALLOC_FAILED ? GBN_ERR_NOMEM : GBN_ERR_CUFFT,
                        "cufftPlanMany (stack z-FFT): error " + std::to_string((int)r));
    it = s->ffts.emplace(C, h).first;
  }
  *plan = it->second;
  return GBN_OK;
}

int exec_z(cufftHandle h, float2* P, int dir, cudaStream_t st) {
  cufftResult r = cufftSetStream(h, st);
  if (r == CUFFT_SUCCESS)
    r = cufftExecC2C(h, reinterpret_cast<cufftComplex*>(P), reinterpret_cast<cufftComplex*>(P), dir);
  if (r != CUFFT_SUCCESS) return stack_fail(GBN_ERR_CUFFT, "cufftExecC2C (stack z-FFT): error " + std::to_string((int)r));
  return GBN_OK;
}

// Whether the forward z transform runs as one kernel: a warp sums n4 terms for 8
// planes at a time, 64 a round.  256 x 256, 8 coils (us, one kernel / three passes): 64
// planes 165 / 502, 90 580 / 814, 55 (radix 1) 328 / 471, 65 507 / 545, 75 693 / 635; 32 x
// 32, one coil: 7 / 13, 15 / 13, 9 / 13, 15 / 12, 17 / 13.
bool fwd_in_one(const gbn_stack_s* s, int C) {
  return s->radix && s->dft.n4 * ((s->dft.npad + 63) / 64) <= (s->g.nxy * C >= 4096 ? 100 : 80);
}

// The same for the adjoint, whose CTAs walk over the coils with maps.  Estimates in us
// with rates measured on 32^2 to 256^2 x 9 to 126 planes and 1, 8 coils: the sum takes
// 0.32 us a million terms, at least 8 ns a CTA and coil, or its chain where few columns
// leave the GPU idle (14 ns a term of a warp, for every coil with maps); the three passes
// 14.5 ps a cell while the stack stays in L2, up to 2.3 times that beyond.  128 x 128, 8
// coils: 64 planes 98 / 127, 120 264 / 298, 45 (radix 1) 139 / 99, 75 332 / 163; 256 x
// 256: 9 planes 121 / 76, 64 351 / 902; 32 x 32 with maps: 64 planes 35 / 21, 75 101 / 25.
bool adj_in_one(const gbn_stack_s* s, int C, bool maps) {
  if (!s->radix) return false;
  const StackGeom& g = s->g;
  const StackDft& d = s->dft;
  const double cols = (double)g.nxy * C, cells = cols * g.nz, kept = cols * g.nzi;
  const double chain = 0.0136 * ((d.n4 + 7) / 8) * d.npad;
  const double lat = 5.5 + (maps ? C * (chain + 1.8) : chain);
  const double sum = 7.0 + 0.32e-6 * cols * d.n4 * d.npad + 3.2e-6 * (cells + kept);
  const double ctas = 7.0 + 0.0078 * cols / kDftCols;
  const double one = maps ? std::fmax(1.13 * sum, 1.25 * ctas) : std::fmax(sum, ctas);
  const double beyond = std::fmin(std::fmax((cells + kept - 20e6) / 45e6, 0.0), 1.3);
  const double three = 13.0 + (1.0 + beyond) * (9e-6 * cells + 5.5e-6 * kept);
  return std::fmax(lat, one) < (maps ? 0.88 : 1.0) * three;
}

// Tables of the one-kernel z transforms when the stack fits them: distinct planes
// (a repeated one is written by an unspecified copy in the scatter) and tables
// and columns within 96 KB of shared memory.
int stack_setup_dft(gbn_stack s, const std::vector<int>& pos) {
  const StackGeom& g = s->g;
  const int R = g.nz % 4 == 0 ? 4 : g.nz % 2 == 0 ? 2 : 1;
  const int n4 = g.nz / R;
  if (n4 > 8 * (16 / R)) return GBN_OK;
  std::vector<char> seen(g.nz, 0);
  std::vector<int> order, freq;
  for (int f : pos) {
    if (seen[f]) return GBN_OK;
    seen[f] = 1;
  }
  for (int r = 0; r < R; ++r) {
    for (size_t k = 0; k < pos.size(); ++k)
      if (pos[k] % R == r) {
        order.push_back((int)k * 4 + r);
        freq.push_back(pos[k]);
      }
    while (order.size() % 8) {
      order.push_back(-4 + r);  // >> 2 is -1, the residue stays in the low bits
      freq.push_back(-1);
    }
  }
  const int npad = (int)order.size();
  const size_t wb = (size_t)n4 * npad * sizeof(float2);
  s->smem_fwd = wb + (size_t)g.nz * (kDftCols + 1) * sizeof(float2);
  s->smem_adj = wb + (size_t)npad * kDftCols * sizeof(float2) + (size_t)kDftCols * (g.nz + 2) * sizeof(float2);
  if (s->smem_fwd > 96 * 1024 || s->smem_adj > 96 * 1024) return GBN_OK;
  std::vector<float2> W((size_t)n4 * npad, make_float2(0.f, 0.f));
  const double pi = 3.14159265358979323846;
  for (int z = 0; z < n4; ++z)
    for (int j = 0; j < npad; ++j)
      if (freq[j] >= 0) {
        const double a = 2.0 * pi * (double)((int64_t)freq[j] * z % g.nz) / g.nz;
        W[(size_t)z * npad + j] = make_float2((float)std::cos(a), (float)-std::sin(a));
      }
  int rc = ck_cuda(cudaMalloc(&s->W, wb), "stack z table");
  if (!rc) rc = ck_cuda(cudaMemcpy(s->W, W.data(), wb, cudaMemcpyHostToDevice), "stack z table");
  if (!rc) rc = ck_cuda(cudaMalloc(&s->order, sizeof(int) * npad), "stack plane order");
  if (!rc)
    rc = ck_cuda(cudaMemcpy(s->order, order.data(), sizeof(int) * npad, cudaMemcpyHostToDevice),
                 "stack plane order");
  for (const void* k : {(const void*)stack_fwd_dft_kernel<1>, (const void*)stack_fwd_dft_kernel<2>,
                        (const void*)stack_fwd_dft_kernel<4>, (const void*)stack_adj_dft_kernel<1>,
                        (const void*)stack_adj_dft_kernel<2>, (const void*)stack_adj_dft_kernel<4>})
    if (!rc)
      rc = ck_cuda(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024),
                   "stack kernel attributes");
  if (rc) return rc;
  s->dft = StackDft{s->W, s->order, n4, npad};
  s->radix = R;
  return GBN_OK;
}

}  // namespace

extern "C" {

int gbn_stack_create(const int64_t* shape, const int* z_index, int n_index, int device,
                     gbn_stack* out) {
  if (!out || !shape || (!z_index && n_index > 0) || n_index < 1)
    return stack_fail(GBN_ERR_ARG, "invalid stack arguments");
  *out = nullptr;
  for (int d = 0; d < 3; ++d)
    if (shape[d] < 1 || shape[d] > (1 << 20)) return stack_fail(GBN_ERR_ARG, "stack shape out of range");
  const int nz = (int)shape[2];
  std::vector<int> pos(n_index);
  for (int k = 0; k < n_index; ++k) {
    if (z_index[k] < 0 || z_index[k] >= nz) return stack_fail(GBN_ERR_ARG, "z_index out of range");
    int p = z_index[k] - nz / 2;  // frequency of the shifted index, as a DFT bin
    pos[k] = p < 0 ? p + nz : p;
  }
  DevSwitch dg(device);
  gbn_stack s = new gbn_stack_s();
  s->device = device;
  s->g.nx = (int)shape[0];
  s->g.ny = (int)shape[1];
  s->g.nz = nz;
  s->g.nzi = n_index;
  s->g.nxy = shape[0] * shape[1];
  s->g.nimg = s->g.nxy * nz;
  int rc = ck_cuda(cudaMalloc(&s->zpos, sizeof(int) * n_index), "stack z positions");
  if (!rc)
    rc = ck_cuda(cudaMemcpy(s->zpos, pos.data(), sizeof(int) * n_index, cudaMemcpyHostToDevice),
                 "stack z positions");
  if (!rc) rc = stack_setup_dft(s, pos);
  if (rc) {
    delete s;
    return rc;
  }
  *out = s;
  return GBN_OK;
}

int gbn_stack_fwd(gbn_stack s, const void* img, const void* smaps, void* out, int C,
                  gbn_stream stream) {
  if (!s || !img || !out || C < 1) return stack_fail(GBN_ERR_ARG, "invalid stack arguments");
  DevSwitch dg(s->device);
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const StackGeom& g = s->g;
  const float scale = (float)(1.0 / std::sqrt(2.0 * g.nz));
  if (C <= 65535 && fwd_in_one(s, C)) {
    const float2 *x = static_cast<const float2*>(img), *m = static_cast<const float2*>(smaps);
    float2* const y = static_cast<float2*>(out);
    return ck_cuda(s->radix == 4   ? dft_fwd<4>(g, s->dft, x, m, y, C, scale, s->smem_fwd, st)
                   : s->radix == 2 ? dft_fwd<2>(g, s->dft, x, m, y, C, scale, s->smem_fwd, st)
                                   : dft_fwd<1>(g, s->dft, x, m, y, C, scale, s->smem_fwd, st),
                   "stack forward");
  }
  cufftHandle h;
  int rc = stack_prepare(s, C, &h);
  if (rc) return rc;
  stack_pad_kernel<<<blocks_for((int64_t)C * g.nimg), 256, 0, st>>>(
      g, static_cast<const float2*>(img), static_cast<const float2*>(smaps), s->P, C);
  if ((rc = ck_cuda(cudaGetLastError(), "stack pad"))) return rc;
  if ((rc = exec_z(h, s->P, CUFFT_FORWARD, st))) return rc;
  stack_gather_kernel<<<blocks_for((int64_t)C * g.nzi * g.nxy), 256, 0, st>>>(
      g, s->P, s->zpos, static_cast<float2*>(out), C, scale);
  return ck_cuda(cudaGetLastError(), "stack gather");
}

int gbn_stack_adj(gbn_stack s, const void* in, const void* smaps, void* img, int C, int accumulate,
                  gbn_stream stream) {
  if (!s || !in || !img || C < 1) return stack_fail(GBN_ERR_ARG, "invalid stack arguments");
  DevSwitch dg(s->device);
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const StackGeom& g = s->g;
  const float scale = (float)(1.0 / std::sqrt(2.0 * g.nz));
  if (C <= 65535 && adj_in_one(s, C, smaps != nullptr)) {
    const float2 *y = static_cast<const float2*>(in), *m = static_cast<const float2*>(smaps);
    float2* const x = static_cast<float2*>(img);
    return ck_cuda(s->radix == 4   ? dft_adj<4>(g, s->dft, y, m, x, C, accumulate, scale, s->smem_adj, st)
                   : s->radix == 2 ? dft_adj<2>(g, s->dft, y, m, x, C, accumulate, scale, s->smem_adj, st)
                                   : dft_adj<1>(g, s->dft, y, m, x, C, accumulate, scale, s->smem_adj, st),
                   "stack adjoint");
  }
  cufftHandle h;
  int rc = stack_prepare(s, C, &h);
  if (rc) return rc;
  if ((rc = ck_cuda(cudaMemsetAsync(s->P, 0, sizeof(float2) * (size_t)C * g.nimg, st), "stack zero")))
    return rc;
  stack_scatter_kernel<<<blocks_for((int64_t)C * g.nzi * g.nxy), 256, 0, st>>>(
      g, static_cast<const float2*>(in), s->zpos, s->P, C, scale);
  if ((rc = ck_cuda(cudaGetLastError(), "stack scatter"))) return rc;
  if ((rc = exec_z(h, s->P, CUFFT_INVERSE, st))) return rc;
  const int64_t n = smaps ? g.nimg : (int64_t)C * g.nimg;
  stack_crop_kernel<<<blocks_for(n), 256, 0, st>>>(g, s->P, static_cast<const float2*>(smaps),
                                                   static_cast<float2*>(img), C, accumulate);
  return ck_cuda(cudaGetLastError(), "stack crop");
}

int gbn_stack_destroy(gbn_stack s) {
  delete s;
  return GBN_OK;
}

}  // extern "C"
