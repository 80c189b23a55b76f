// Pruned 3D transforms on fine grids of 128, 192 or 256 cells an axis, fused with
// the pad and crop passes.
//
// The image modes of an n-point axis occupy the fine indices [0, n - n/2) and
// [nf - n/2, nf).  A type-2 transform (op) therefore starts from a grid that is
// non-zero only on the (x mode, y mode, z mode) cells, and a type-1 transform
// (adjoint) keeps only those cells of its result.  The library's cuFFT path
// writes every fine cell in the pad pass and runs full 2D transforms over the
// mode planes, then 1D transforms along x.  Here each axis is a separate pass of
// line transforms that reads only the lines and entries that can be non-zero and
// writes only the entries that a later pass reads:
//
//   op      z lines of the (x mode, y mode) columns, pad fused into the
//           loads (x * s * scale / phihat), the z modes of a line;
//           y lines of the x-mode planes (mode entries in, all out);
//           x lines of every (y, z) (mode entries in, all out).
//   adjoint x lines of every (y, z) (all in, mode entries out);
//           y lines of the x-mode planes (all in, mode entries out);
//           z lines of the (x mode, y mode) columns (all in, mode entries
//           out), crop fused into the stores (divide by phihat, scale, and
//           the SENSE coil combine sum_c conj(s_c) v_c over the pass's coils).
//   Toeplitz Gram (256-point x axis): the op's z and y passes, one pass over the
//           (y, z) lines doing the forward x transform, the multiply by the
//           spectrum and the inverse x transform, then the adjoint's y and z
//           passes.
//
// For a 128^3 image on 256^3 cells this moves about 350 MB per coil and
// transform against about 670 MB for the pad pass plus the pruned cuFFT passes.
// Where the image has half as many modes as the axis has cells, the entries of a
// line that hold modes are whole rows of the four-step layout, a compile-time set
// (kHalf); other sizes test each entry at run time (kModes).
//
// A line of 16 A cells (A = 8, 12, 16) is an A-point and a 16-point DFT in
// registers with one exchange through shared memory (four-step: n = 16 a + b,
// k = k1 + A k2):
//   Y_b[k1] = sum_a x[16 a + b] W_A^(a k1),   Z_b[k1] = Y_b[k1] W_N^(b k1),
//   X[k1 + A k2] = sum_b Z_b[k1] W16^(b k2).
// A thread owns one (line, b) in the first step and one (line, k1 < A) in the
// second.  The exponent sign is -1; a +1 transform conjugates its inputs and
// outputs.  The twiddles W_N^(b k1) come from a table computed in double
// precision on the host, laid out [k1][b] so that lanes running over b read
// consecutive entries.
//
// Against cuFFT with pad and crop: 96^3 images (192^3 cells), 8 coils, op + adj
// 1.04 -> 0.48 ms.
//
// Thread layouts (256 threads, 16 lines per CTA):
//   z lines (contiguous in memory): lanes run over b (first step) or k1
//     (second step) of two lines, so each global access is a 128-byte row
//     segment; the exchange buffer [line][k1][b] has a row pitch of 17
//     cells, which keeps both steps free of bank conflicts;
//   x / y lines: lanes run over 16 consecutive z columns, so each global access
//     is again a 128-byte segment; the exchange buffer is [k1][b][z].
#include "gbn_fft3d.cuh"
#include "gbn_dft.cuh"

#include <cmath>
#include <vector>

namespace gbn {

namespace {

using namespace dft;

constexpr int kLines = 16;       // lines per CTA
constexpr int kThreads = 256;

__device__ __forceinline__ int img_to_fine(int i, int n, int nf) {
  const int k = i - (n >> 1);
  return k < 0 ? k + nf : k;
}

// Entry m = 16 q + b of a line of 16 A cells, for the mode sets of the
// transformed axis: kAll (every entry), kHalf (n = 8 A: the modes are the rows
// q < A / 4 and q >= 3 A / 4, known at compile time in the unrolled loops),
// kModes (any n <= 16 A; the upper half of a line can only hold negative modes,
// so the test and the image index differ by row at compile time).  In the
// outputs' order m = k1 + A k2 the same with k2 < 4 and k2 >= 12, or k2 < 8.
enum : int { kAll = 0, kHalf = 1, kModes = 2 };
template <int A, int SET>
__device__ __forceinline__ bool in_on(int q, int b, int n) {
  if (SET == kAll) return true;
  if (SET == kHalf) return q < A / 4 || q >= 3 * A / 4;
  const int m = 16 * q + b;
  return q < A / 2 ? m < n - (n >> 1) : m >= 16 * A - (n >> 1);
}
template <int A, int SET>
__device__ __forceinline__ int in_img(int q, int b, int n) {  // image index of a mode entry
  if (SET == kHalf) return 16 * q + b + (q < A / 4 ? 4 * A : -12 * A);
  return 16 * q + b + (n >> 1) - (q < A / 2 ? 0 : 16 * A);
}
template <int A, int SET>
__device__ __forceinline__ bool out_on(int k2, int k1, int n) {
  if (SET == kAll) return true;
  if (SET == kHalf) return k2 < 4 || k2 >= 12;
  const int m = k1 + A * k2;
  return k2 < 8 ? m < n - (n >> 1) : m >= 16 * A - (n >> 1);
}
template <int A, int SET>
__device__ __forceinline__ int out_img(int k2, int k1, int n) {
  if (SET == kHalf) return k1 + A * k2 + (k2 < 4 ? 4 * A : -12 * A);
  return k1 + A * k2 + (n >> 1) - (k2 < 8 ? 0 : 16 * A);
}

// The twiddle table goes through a register and is stored after the line's loads
// are under way: a store (or a branch) before them makes them wait for the table
// (pad 45 against 56 us for 4 coils of 128^3 images).
template <int N>
__device__ __forceinline__ float2 tw_load(const float2* __restrict__ tw) {
  return tw[N == kThreads ? threadIdx.x : threadIdx.x % N];
}
template <int N>
__device__ __forceinline__ void tw_store(float2* s_tw, float2 v) {
  s_tw[N == kThreads ? threadIdx.x : threadIdx.x % N] = v;  // the same value where entries repeat
}

// first step: the A-point DFT of the first A of a thread's 16 entries; its output
// k1 is first_out<A>(x, k1)
template <int A, bool HALF_IN = false>
__device__ __forceinline__ void first_step(float2 (&x)[16]) {
  dftn<A, HALF_IN, false>(*reinterpret_cast<float2(*)[A]>(x));
}
template <int A>
__device__ __forceinline__ float2 first_out(const float2 (&x)[16], int k1) {
  return x[dftn_pos<A>(k1)];
}

// ---------------------------------------------------------------- z lines, pad fused
// blockIdx.x: 16 consecutive (ix, iy) image columns; blockIdx.y: transform;
// SET: the z modes
template <int A, int SET>
__global__ void __launch_bounds__(kThreads)
f3_pad_z_kernel(PadArgs a, const float2* __restrict__ tw, int conj) {
  constexpr int N = 16 * A;
  __shared__ float2 s_tw[N];
  __shared__ float2 s_x[kLines * A * 17];
  const Geom& g = a.g;
  const int n0 = g.n[0], n1 = g.n[1], n2 = g.n[2];
  const float2 twv = tw_load<N>(tw);
  const int b = threadIdx.x & 15, l = threadIdx.x >> 4;
  const int line = blockIdx.x * kLines + l;
  const bool valid = line < n0 * n1;
  const int ix = valid ? line / n1 : 0, iy = valid ? line - ix * n1 : 0;
  const int c = blockIdx.y;
  const int64_t irow = ((int64_t)ix * n1 + iy) * n2;
  const float2* img = a.smaps ? a.img : a.img + (int64_t)c * g.Nimg;
  const float2* sm = a.smaps ? a.smaps + (int64_t)c * g.Nimg : nullptr;
  float f0 = a.scale;
  if (a.dec[0]) f0 *= a.dec[0][ix];
  if (a.dec[1]) f0 *= a.dec[1][iy];
  float2 x[16];
#pragma unroll
  for (int q = 0; q < A; ++q) {
    float2 v = make_float2(0.f, 0.f);
    if (valid && in_on<A, SET>(q, b, n2)) {
      const int i2 = in_img<A, SET>(q, b, n2);
      v = img[irow + i2];
      if (a.conj_in) v = f2conj(v);
      if (sm) {
        float2 s = sm[irow + i2];
        if (a.conj_in) s = f2conj(s);
        v = f2mul(v, s);
      }
      v = f2scale(v, a.dec[2] ? f0 * a.dec[2][i2] : f0);
      if (conj) v = f2conj(v);
    }
    x[q] = v;
  }
  tw_store<N>(s_tw, twv);
  __syncthreads();  // twiddle table
  first_step<A, SET == kHalf>(x);
  float2* row = s_x + l * (A * 17);
#pragma unroll
  for (int k1 = 0; k1 < A; ++k1) row[k1 * 17 + b] = f2mul(first_out<A>(x, k1), s_tw[k1 * 16 + b]);
  __syncthreads();
  const int k1 = b;
  if (A < 16 && k1 >= A) return;
#pragma unroll
  for (int q = 0; q < 16; ++q) x[q] = row[k1 * 17 + q];
  dft16(x);
  if (!valid) return;
  float2* out = a.fine + (int64_t)c * g.G +
                ((int64_t)img_to_fine(ix, n0, g.nf[0]) * g.nf[1] + img_to_fine(iy, n1, g.nf[1])) * N + k1;
#pragma unroll
  for (int k2 = 0; k2 < 16; ++k2) {
    const float2 v = x[pos16(k2)];
    out[A * k2] = conj ? f2conj(v) : v;
  }
}

// ---------------------------------------------------------------- x / y lines
struct Lines3 {
  float2* data;       // ntr grids of G cells
  int64_t G;
  int64_t line_stride;   // cells between consecutive entries of a line
  int64_t outer_stride;  // cells between consecutive outer indices
  int outer_modes;       // outer index o is an image index of an n_outer-point axis of nf_outer cells
  int n_outer, nf_outer;
  int n_axis;            // image size along the transformed axis
  int in_prune;          // only mode entries are read (the others are zero)
  int out_prune;         // only mode entries are written
  int conj;
  const float2* tw;
};

// blockIdx.x: 16 consecutive z columns; blockIdx.y: outer index; blockIdx.z: transform
// IN / OUT: the entries read / written (kAll, kHalf, kModes of n_axis)
template <int A, int MINB, int IN, int OUT>
__global__ void __launch_bounds__(kThreads, MINB) f3_lines_kernel(Lines3 a) {
  constexpr int N = 16 * A;
  __shared__ float2 s_tw[N];
  __shared__ float2 s_x[A * 16 * kLines];
  const float2 twv = tw_load<N>(a.tw);
  const int l = threadIdx.x & 15, b = threadIdx.x >> 4;
  const int z = blockIdx.x * kLines + l;
  const int o = a.outer_modes ? img_to_fine(blockIdx.y, a.n_outer, a.nf_outer) : (int)blockIdx.y;
  float2* base = a.data + (int64_t)blockIdx.z * a.G + o * a.outer_stride + z;
  float2 x[16];
#pragma unroll
  for (int q = 0; q < A; ++q) {
    float2 v = make_float2(0.f, 0.f);
    if (in_on<A, IN>(q, b, a.n_axis)) {
      v = base[(16 * q + b) * a.line_stride];
      if (a.conj) v = f2conj(v);
    }
    x[q] = v;
  }
  tw_store<N>(s_tw, twv);
  __syncthreads();  // twiddle table
  first_step<A, IN == kHalf>(x);
#pragma unroll
  for (int k1 = 0; k1 < A; ++k1) s_x[(k1 * 16 + b) * 16 + l] = f2mul(first_out<A>(x, k1), s_tw[k1 * 16 + b]);
  __syncthreads();
  const int k1 = b;
  if (k1 >= A) return;
#pragma unroll
  for (int q = 0; q < 16; ++q) x[q] = s_x[(k1 * 16 + q) * 16 + l];
  dft16<false, OUT == kHalf>(x);
#pragma unroll
  for (int k2 = 0; k2 < 16; ++k2) {
    if (out_on<A, OUT>(k2, k1, a.n_axis)) {
      const float2 v = x[pos16(k2)];
      base[(k1 + A * k2) * a.line_stride] = a.conj ? f2conj(v) : v;
    }
  }
}

// ---------------------------------------------------------------- z lines, crop fused
// blockIdx.x: 16 consecutive (ix, iy) image columns; the CTA runs every
// transform of the pass and, with coil maps, sums them into one image
template <int A>
constexpr size_t crop_smem() {
  return (16 * A + kLines * A * 17 + kLines * A * 16) * sizeof(float2);
}

template <int A, int MINB, int SET>
__global__ void __launch_bounds__(kThreads, MINB)
f3_z_crop_kernel(CropArgs a, const float2* __restrict__ tw, int conj) {
  constexpr int N = 16 * A;
  // dynamic: twiddles, the exchange buffer, and the coil sums [line][k2][k1]
  // (thread (line, k1) owns its 16 entries)
  extern __shared__ float2 s_dyn[];
  float2* const s_tw = s_dyn;
  float2* const s_x = s_tw + N;
  float2* const s_acc = s_x + kLines * A * 17;
  const Geom& g = a.g;
  const int n0 = g.n[0], n1 = g.n[1], n2 = g.n[2];
  tw_store<N>(s_tw, tw_load<N>(tw));
  const int b = threadIdx.x & 15, l = threadIdx.x >> 4;
  const int line = blockIdx.x * kLines + l;
  const bool valid = line < n0 * n1;
  const int ix = valid ? line / n1 : 0, iy = valid ? line - ix * n1 : 0;
  const int64_t irow = ((int64_t)ix * n1 + iy) * n2;
  const int64_t frow =
      ((int64_t)img_to_fine(ix, n0, g.nf[0]) * g.nf[1] + img_to_fine(iy, n1, g.nf[1])) * N;
  float f0 = a.scale;
  if (a.dec[0]) f0 *= a.dec[0][ix];
  if (a.dec[1]) f0 *= a.dec[1][iy];
  float2* row = s_x + l * (A * 17);
  const int k1 = b;
  float2* acc = s_acc + l * N + k1;      // entry k2 at acc[A * k2]
  if (A == 16 || k1 < A) {
#pragma unroll
    for (int k2 = 0; k2 < 16; ++k2) acc[A * k2] = make_float2(0.f, 0.f);
  }
  for (int c = 0; c < a.ntr; ++c) {
    const float2* in = a.fine + (int64_t)c * g.G + frow;
    float2 x[16];
#pragma unroll
    for (int q = 0; q < A; ++q) {
      float2 v = valid ? in[16 * q + b] : make_float2(0.f, 0.f);
      x[q] = conj ? f2conj(v) : v;
    }
    float2 s8[8];  // kHalf: the coil map's entries, loaded with the line
    if (SET == kHalf && a.smaps && valid && (A == 16 || k1 < A)) {
      const float2* sm = a.smaps + (int64_t)c * g.Nimg + irow + k1;
#pragma unroll
      for (int k = 0; k < 8; ++k) s8[k] = sm[A * k];
    }
    __syncthreads();  // twiddle table; the previous transform's exchange reads are done
    first_step<A>(x);
#pragma unroll
    for (int kk = 0; kk < A; ++kk) row[kk * 17 + b] = f2mul(first_out<A>(x, kk), s_tw[kk * 16 + b]);
    __syncthreads();
    if (A < 16 && k1 >= A) continue;
#pragma unroll
    for (int q = 0; q < 16; ++q) x[q] = row[k1 * 17 + q];
    dft16<false, SET == kHalf>(x);
    if (!valid) continue;
#pragma unroll
    for (int k2 = 0; k2 < 16; ++k2) {
      if (!out_on<A, SET>(k2, k1, n2)) continue;
      const int i2 = out_img<A, SET>(k2, k1, n2);
      float2 v = x[pos16(k2)];
      if (conj) v = f2conj(v);
      if (a.smaps) {
        const float2 s =
            SET == kHalf ? s8[(k2 + 4) & 7] : a.smaps[(int64_t)c * g.Nimg + irow + i2];
        const float2 o = acc[A * k2];
        acc[A * k2] = make_float2(o.x + s.x * v.x + s.y * v.y, o.y + s.x * v.y - s.y * v.x);
      } else {
        const float f = a.dec[2] ? f0 * a.dec[2][i2] : f0;
        float2 r = f2scale(v, f);
        float2* dst = a.out + (int64_t)c * g.Nimg + irow + i2;
        if (a.accumulate) r = f2add(r, *dst);
        *dst = r;
      }
    }
  }
  if (!a.smaps || !valid || (A < 16 && k1 >= A)) return;
#pragma unroll
  for (int k2 = 0; k2 < 16; ++k2) {
    if (!out_on<A, SET>(k2, k1, n2)) continue;
    const int i2 = out_img<A, SET>(k2, k1, n2);
    const float f = a.dec[2] ? f0 * a.dec[2][i2] : f0;
    float2 r = f2scale(acc[A * k2], f);
    float2* dst = a.out + irow + i2;
    if (a.accumulate) r = f2add(r, *dst);
    *dst = r;
  }
}

// ---------------------------------------------------------------- x lines of the Toeplitz Gram
// 256-point x axis.  Forward x transform (x-mode entries in), multiply by the real kernel K,
// inverse x transform (x-mode entries out) of every (y, z) line, for every
// transform of the pass, without writing the full grid.  After the forward
// transform's second step thread (z, k1) holds X[k1 + 16 k2], k2 = 0 .. 15,
// which are exactly the inputs x[16 a + b] (a = k2) of the inverse
// transform's first step for b = k1, so the two transforms share one layout.
// blockIdx.x: 16 consecutive z columns; blockIdx.y: y.  CUBE: 256 cells on every
// axis (the x stride as a constant saves registers)
template <int SET, bool CUBE>
__global__ void __launch_bounds__(kThreads, 4)
f3_x_kmul_kernel(float2* data, int64_t G, int nf1, int nf2, int ntr, int n0, const float* __restrict__ K,
                 const float2* __restrict__ tw) {
  const int64_t XS = CUBE ? 256 * 256 : (int64_t)nf1 * nf2;  // x stride
  __shared__ float2 s_tw[256];
  __shared__ float2 s_x[16 * 16 * kLines];
  s_tw[threadIdx.x] = tw[threadIdx.x];
  const int l = threadIdx.x & 15, b = threadIdx.x >> 4;
  const int z = blockIdx.x * kLines + l;
  const int64_t col = (int64_t)blockIdx.y * (CUBE ? 256 : nf2) + z;
  float kk[16];  // K at x = b + 16 k2 (b is k1 in the forward transform's second step)
#pragma unroll
  for (int k2 = 0; k2 < 16; ++k2) kk[k2] = K[(b + 16 * k2) * XS + col];
  for (int c = 0; c < ntr; ++c) {
    float2* base = data + (int64_t)c * G + col;
    float2 x[16];
#pragma unroll
    for (int q = 0; q < 16; ++q)
      x[q] = in_on<16, SET>(q, b, n0) ? base[(16 * q + b) * XS] : make_float2(0.f, 0.f);
    __syncthreads();  // twiddles; the previous transform's exchange reads are done
    dft16<SET == kHalf>(x);
#pragma unroll
    for (int k1 = 0; k1 < 16; ++k1) s_x[(k1 * 16 + b) * 16 + l] = f2mul(x[pos16(k1)], s_tw[k1 * 16 + b]);
    __syncthreads();
    // thread (z, k1 = b): X[k1 + 16 k2] -> conj(K X) as the inverse transform's x[16 k2 + k1]
    float2 y[16];
#pragma unroll
    for (int q = 0; q < 16; ++q) y[q] = s_x[(b * 16 + q) * 16 + l];
    dft16(y);
#pragma unroll
    for (int k2 = 0; k2 < 16; ++k2) x[k2] = f2conj(f2scale(y[pos16(k2)], kk[k2]));
    dft16(x);
    __syncthreads();  // every thread has read its forward exchange entries
#pragma unroll
    for (int k1 = 0; k1 < 16; ++k1) s_x[(k1 * 16 + b) * 16 + l] = f2mul(x[pos16(k1)], s_tw[k1 * 16 + b]);
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 16; ++q) y[q] = s_x[(b * 16 + q) * 16 + l];
    dft16<false, SET == kHalf>(y);
#pragma unroll
    for (int k2 = 0; k2 < 16; ++k2)
      if (out_on<16, SET>(k2, b, n0)) base[(b + 16 * k2) * XS] = f2conj(y[pos16(k2)]);
  }
}

}  // namespace

bool fft3d_fits(const Geom& g) {
  if (g.dim != 3) return false;
  for (int d = 0; d < 3; ++d)
    if (g.nf[d] != 128 && g.nf[d] != 192 && g.nf[d] != 256) return false;
  return true;
}

std::vector<float> fft_twiddles(int n) {
  // entry k1 * 16 + b (k1 < n / 16): W_n^(b k1) = exp(-2 pi i b k1 / n), as (re, im)
  std::vector<float> t(2 * n);
  const double pi = 3.14159265358979323846;
  for (int k1 = 0; k1 < n / 16; ++k1)
    for (int b = 0; b < 16; ++b) {
      const int e = k1 * 16 + b;
      t[2 * e] = (float)std::cos(2.0 * pi * b * k1 / n);
      t[2 * e + 1] = (float)-std::sin(2.0 * pi * b * k1 / n);
    }
  return t;
}

namespace {

template <int A>
void lines_a(const Lines3& a, dim3 grid, cudaStream_t st) {
  // 256 points: 4 CTAs per SM (64 registers, a few bytes of spills) measured 5 %
  // faster than 3 CTAs at 80 registers on the 128^3 passes
  const bool half = a.n_axis == 8 * A;
  if (a.in_prune) {
    if (half) f3_lines_kernel<A, 4, kHalf, kAll><<<grid, kThreads, 0, st>>>(a);
    else f3_lines_kernel<A, 4, kModes, kAll><<<grid, kThreads, 0, st>>>(a);
  } else {
    if (half) f3_lines_kernel<A, 4, kAll, kHalf><<<grid, kThreads, 0, st>>>(a);
    else f3_lines_kernel<A, 4, kAll, kModes><<<grid, kThreads, 0, st>>>(a);
  }
}
void lines(const Lines3& a, int nf, dim3 grid, cudaStream_t st) {
  if (nf == 256) lines_a<16>(a, grid, st);
  else if (nf == 192) lines_a<12>(a, grid, st);
  else lines_a<8>(a, grid, st);
}

template <int A>
void pad_z_a(const PadArgs& pa, const float2* tw, int conj, cudaStream_t st) {
  const int nl = pa.g.n[0] * pa.g.n[1];
  const dim3 grid((nl + kLines - 1) / kLines, pa.ntr);
  if (pa.g.n[2] == 8 * A) f3_pad_z_kernel<A, kHalf><<<grid, kThreads, 0, st>>>(pa, tw, conj);
  else f3_pad_z_kernel<A, kModes><<<grid, kThreads, 0, st>>>(pa, tw, conj);
}
void pad_z(const PadArgs& pa, const Twiddles& tw, int conj, cudaStream_t st) {
  if (pa.g.nf[2] == 256) pad_z_a<16>(pa, tw.t[2], conj, st);
  else if (pa.g.nf[2] == 192) pad_z_a<12>(pa, tw.t[2], conj, st);
  else pad_z_a<8>(pa, tw.t[2], conj, st);
}

// coil sums in shared memory: 3 CTAs per SM (69 against 86 us with the sums
// in registers at 2 CTAs per SM, 4 coils of a 128^3 image).  Half-size axes take
// the instance that loads the map's 8 entries with the line, before the first
// wait: 67 -> 51 us (218 MB, 4.3 TB/s) against loading them after the transform.
template <int A>
void z_crop_a(const CropArgs& ca, const float2* tw, int conj, cudaStream_t st) {
  const int nl = ca.g.n[0] * ca.g.n[1];
  const unsigned nb = (nl + kLines - 1) / kLines;
  auto k = ca.g.n[2] == 8 * A ? f3_z_crop_kernel<A, 3, kHalf> : f3_z_crop_kernel<A, 3, kModes>;
  k<<<nb, kThreads, crop_smem<A>(), st>>>(ca, tw, conj);
}
cudaError_t z_crop(const CropArgs& ca, const Twiddles& tw, int conj, cudaStream_t st) {
  if (ca.g.nf[2] == 256) z_crop_a<16>(ca, tw.t[2], conj, st);
  else if (ca.g.nf[2] == 192) z_crop_a<12>(ca, tw.t[2], conj, st);
  else z_crop_a<8>(ca, tw.t[2], conj, st);
  return cudaGetLastError();
}

void y_lines(float2* fine, const Geom& g, const Twiddles& tw, int ntr, int in_prune, int conj, cudaStream_t st) {
  Lines3 y{};
  y.data = fine;
  y.G = g.G;
  y.line_stride = g.nf[2];
  y.outer_stride = (int64_t)g.nf[1] * g.nf[2];
  y.outer_modes = 1;
  y.n_outer = g.n[0];
  y.nf_outer = g.nf[0];
  y.n_axis = g.n[1];
  y.in_prune = in_prune;
  y.out_prune = !in_prune;
  y.conj = conj;
  y.tw = tw.t[1];
  lines(y, g.nf[1], dim3(g.nf[2] / kLines, g.n[0], ntr), st);
}

void x_lines(float2* fine, const Geom& g, const Twiddles& tw, int ntr, int in_prune, int conj, cudaStream_t st) {
  Lines3 x{};
  x.data = fine;
  x.G = g.G;
  x.line_stride = (int64_t)g.nf[1] * g.nf[2];
  x.outer_stride = g.nf[2];
  x.outer_modes = 0;
  x.n_axis = g.n[0];
  x.in_prune = in_prune;
  x.out_prune = !in_prune;
  x.conj = conj;
  x.tw = tw.t[0];
  lines(x, g.nf[0], dim3(g.nf[2] / kLines, g.nf[1], ntr), st);
}
}  // namespace

cudaError_t fft3d_prepare() {
  auto set = [](auto k, size_t b) {
    return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)b);
  };
  cudaError_t e = set(f3_z_crop_kernel<16, 3, kModes>, crop_smem<16>());
  if (e == cudaSuccess) e = set(f3_z_crop_kernel<12, 3, kModes>, crop_smem<12>());
  if (e == cudaSuccess) e = set(f3_z_crop_kernel<8, 3, kModes>, crop_smem<8>());
  if (e == cudaSuccess) e = set(f3_z_crop_kernel<16, 3, kHalf>, crop_smem<16>());
  if (e == cudaSuccess) e = set(f3_z_crop_kernel<12, 3, kHalf>, crop_smem<12>());
  if (e == cudaSuccess) e = set(f3_z_crop_kernel<8, 3, kHalf>, crop_smem<8>());
  return e;
}

cudaError_t launch_fft3d_op(const PadArgs& pa, const Twiddles& tw, int isign, cudaStream_t st) {
  const int conj = isign > 0;
  pad_z(pa, tw, conj, st);
  y_lines(pa.fine, pa.g, tw, pa.ntr, 1, conj, st);
  x_lines(pa.fine, pa.g, tw, pa.ntr, 1, conj, st);
  return cudaGetLastError();
}

cudaError_t launch_fft3d_adj(const CropArgs& ca, float2* fine, const Twiddles& tw, int isign,
                             cudaStream_t st) {
  const int conj = isign > 0;
  x_lines(fine, ca.g, tw, ca.ntr, 0, conj, st);
  y_lines(fine, ca.g, tw, ca.ntr, 0, conj, st);
  return z_crop(ca, tw, conj, st);
}

cudaError_t launch_fft3d_gram(const PadArgs& pa, const CropArgs& ca, const float* K,
                              const Twiddles& tw, cudaStream_t st) {
  const Geom& g = pa.g;
  if (g.nf[0] != 256) return cudaErrorInvalidValue;
  pad_z(pa, tw, 0, st);
  y_lines(pa.fine, g, tw, pa.ntr, 1, 0, st);
  const dim3 grid(g.nf[2] / kLines, g.nf[1]);
  const bool half = g.n[0] == 128, cube = g.nf[1] == 256 && g.nf[2] == 256;
  auto k = half ? (cube ? f3_x_kmul_kernel<kHalf, true> : f3_x_kmul_kernel<kHalf, false>)
                : (cube ? f3_x_kmul_kernel<kModes, true> : f3_x_kmul_kernel<kModes, false>);
  k<<<grid, kThreads, 0, st>>>(pa.fine, g.G, g.nf[1], g.nf[2], pa.ntr, g.n[0], K, tw.t[0]);
  y_lines(pa.fine, g, tw, pa.ntr, 0, 1, st);
  return z_crop(ca, tw, 1, st);
}

}  // namespace gbn
