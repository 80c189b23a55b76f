// Pruned 2D transforms on fine grids of 256, 384, 512, 640 or 768 cells an axis,
// fused with the pad and crop passes.  The 3D counterpart is gbn_fft3d.cu; the
// layouts below follow it.
//
// Axis 1 (y) is contiguous.  The image modes of an n-point axis occupy the fine
// indices [0, n - n/2) and [nf - n/2, nf).
//
//   op      y lines of the x-mode rows, pad fused into the loads
//           (x * s * scale / phihat on the y modes), all entries
//           written; x lines of every y (mode entries in, all out).
//   adjoint x lines of every y (all in, mode entries out); y lines of the
//           x-mode rows (all in), crop fused into the stores: divide by
//           phihat, scale, and for coil maps conj(s_c) v_c: one coil straight
//           to the image, several added to it with float2 atomics (the image
//           is cleared first unless the call accumulates) or, where the call
//           wants the same bits every time (ordered), left in the rows of the
//           transform's own grid and summed in order by a pass of its own.
//   Toeplitz Gram (512-point x axis): the op's y pass, one pass over the x lines
//           doing the forward transform, the multiply by the real spectrum and
//           the inverse transform, then the adjoint's y pass with the crop.
//
// A line of N = 16 A cells (A = 16, 24, 32, 40, 48) is a four-step of an A-point
// and a 16-point DFT in registers with one exchange through shared memory:
//   n = 16 a + b (a < A, b < 16), k = k1 + A k2 (k1 < A, k2 < 16),
//   Y_b[k1] = sum_a x[16 a + b] W_A^(a k1),   Z_b[k1] = Y_b[k1] W_N^(b k1),
//   X[k1 + A k2] = sum_b Z_b[k1] W16^(b k2).
// A thread owns one (line, b) in the first step and the (line, k1 = b, b + 16, ..)
// of the second.  Where the image has half as many modes as the axis has cells,
// the mode entries of a line are the rows a < A / 4 and a >= 3 A / 4 and the
// outputs k2 < 4 and k2 >= 12, known at compile time (kHalf); other sizes test
// each entry at run time (kModes).
// After the forward 512-point transform's second step the thread (line, b) holds
// X[b + 16 h + 32 k2] (h < 2, k2 < 16), which are the inputs x[16 a' + b]
// (a' = h + 2 k2) of the next 512-point transform's first step: the Gram's
// inverse transform needs no exchange in between.
//
// Against cuFFT with pad and crop: 384^2 images (768^2 cells), 16 coils, op + adj
// 241 -> 138 us.
//
// Thread layouts (256 threads, 16 lines per CTA): y lines put lanes on b of
// two lines (128-byte row segments; exchange buffer [line][k1][b], row
// pitch 17); x lines put lanes on 16 consecutive y columns (exchange buffer
// [k1][b][y]).
#include "gbn_fft2d.cuh"

#include <type_traits>

#include "gbn_dft.cuh"

namespace gbn {

namespace {

using namespace dft;

constexpr int kL = 16;     // lines per CTA
constexpr int kT = 256;    // threads per CTA

// W32^k = (cos(pi k / 16), -sin(pi k / 16)), k < 16
__device__ __forceinline__ float2 w32(int k) {
  constexpr float c[9] = {1.0f,
                          0.98078528040323044f,
                          0.92387953251128674f,
                          0.83146961230254524f,
                          0.70710678118654752f,
                          0.55557023301960218f,
                          0.38268343236508977f,
                          0.19509032201612825f,
                          0.0f};
  return k <= 8 ? make_float2(c[k], -c[8 - k]) : make_float2(-c[16 - k], -c[k - 8]);
}

// 32-point DFT, natural order in and out.  HALF_IN: x[8 .. 23] are zero and
// not read.
template <bool HALF_IN = false>
__device__ __forceinline__ void dft32(float2 (&x)[32]) {
  float2 e[16], o[16];
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    e[j] = x[2 * j];
    o[j] = x[2 * j + 1];
  }
  dft16<HALF_IN>(e);
  dft16<HALF_IN>(o);
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    const float2 ev = e[pos16(k)];
    const float2 ov = f2mul(o[pos16(k)], w32(k));
    x[k] = f2add(ev, ov);
    x[k + 16] = f2sub(ev, ov);
  }
}

// first step of a line; its output k1 is first_out<A>(x, k1)
template <int A, bool HALF_IN = false>
__device__ __forceinline__ void dft_first(float2 (&x)[A]) {
  if constexpr (A == 32) dft32<HALF_IN>(x);
  else dftn<A, HALF_IN, false>(x);
}
template <int A>
__device__ __forceinline__ float2 first_out(const float2 (&x)[A], int k1) {
  return x[A == 32 ? k1 : dftn_pos<A>(k1)];
}

__device__ __forceinline__ bool is_mode(int m, int n, int nf) {
  const int h = n >> 1;
  return m < n - h || m >= nf - h;
}
__device__ __forceinline__ int mode_to_img(int m, int n, int nf) {
  const int h = n >> 1;
  return m < n - h ? m + h : m - nf + h;
}
__device__ __forceinline__ int img_to_fine(int i, int n, int nf) {
  const int k = i - (n >> 1);
  return k < 0 ? k + nf : k;
}

enum : int { kAll = 0, kHalf = 1, kModes = 2 };
// input entry n = 16 a + b
template <int A, int SET>
__device__ __forceinline__ bool in_on(int a, int b, int n) {
  if (SET == kAll) return true;
  if (SET == kHalf) return a < A / 4 || a >= 3 * A / 4;
  return is_mode(16 * a + b, n, 16 * A);
}
template <int A, int SET>
__device__ __forceinline__ int in_img(int a, int b, int n) {  // image index of a mode entry
  if (SET == kHalf) return 16 * a + b + (a < A / 4 ? 4 * A : -12 * A);
  return mode_to_img(16 * a + b, n, 16 * A);
}
// output entry k = k1 + A k2
template <int A, int SET>
__device__ __forceinline__ bool out_on(int k1, int k2, int n) {
  if (SET == kAll) return true;
  if (SET == kHalf) return k2 < 4 || k2 >= 12;
  return is_mode(k1 + A * k2, n, 16 * A);
}

// dynamic shared memory: twiddles + exchange
template <int A>
constexpr size_t y_smem() {
  return (16 * A + kL * A * 17) * sizeof(float2);
}
template <int A>
constexpr size_t x_smem() {
  return (16 * A + A * 16 * kL) * sizeof(float2);
}
// The twiddle table goes through registers and is stored after the line's loads are
// under way, which would wait for a store (or a loop) before them.
template <int A>
struct TwRegs {
  static constexpr int kPer = (16 * A + kT - 1) / kT;
  float2 v[kPer];
  __device__ __forceinline__ explicit TwRegs(const float2* __restrict__ tw) {
#pragma unroll
    for (int i = 0; i < kPer; ++i) v[i] = tw[index(i)];
  }
  __device__ __forceinline__ void store(float2* s_tw) const {
#pragma unroll
    for (int i = 0; i < kPer; ++i) s_tw[index(i)] = v[i];
  }
  // the last round wraps where 16 A is no multiple of the threads: the same values again
  static __device__ __forceinline__ int index(int i) {
    const int e = threadIdx.x + i * kT;
    return 16 * A % kT == 0 ? e : e % (16 * A);
  }
};
// resident CTAs: 3 for the pad of up to 512 points (80 registers: 23.5 against
// 26.9 us at 2 CTAs and 126 registers for 64 transforms), 2 otherwise (the other
// kernels measured slower at 3), 1 where 40 or 48 entries and their exchange need it
template <int A>
constexpr int kPadCtas = A <= 32 ? 3 : 1;
template <int A>
constexpr int kCtas = A <= 32 ? 2 : 1;

// ---------------------------------------------------------------- y lines, pad fused
// blockIdx.x: 16 consecutive x image rows; blockIdx.y: transform.  SET: the y modes.
template <int A, int SET>
__global__ void __launch_bounds__(kT, kPadCtas<A>)
f2_pad_y_kernel(PadArgs a, const float2* __restrict__ tw, int conj) {
  extern __shared__ float2 s_dyn[];
  float2* const s_tw = s_dyn;
  float2* const s_x = s_tw + 16 * A;
  const Geom& g = a.g;
  const int n0 = g.n[0], n1 = g.n[1];
  const TwRegs<A> twv(tw);
  const int b = threadIdx.x & 15, l = threadIdx.x >> 4;
  const int ix = blockIdx.x * kL + l;
  const bool valid = ix < n0;
  const int c = blockIdx.y;
  const int64_t irow = (int64_t)(valid ? ix : 0) * n1;
  const float2* img = a.smaps ? a.img : a.img + (int64_t)c * g.Nimg;
  const float2* sm = a.smaps ? a.smaps + (int64_t)c * g.Nimg : nullptr;
  float f0 = a.scale;
  if (a.dec[0]) f0 *= a.dec[0][valid ? ix : 0];
  if (a.fmax && blockIdx.x == 0 && threadIdx.x == 0) a.fmax[c] = 0;  // the x pass comes after
  float2 x[A];
#pragma unroll
  for (int q = 0; q < A; ++q) {
    float2 v = make_float2(0.f, 0.f);
    if (valid && in_on<A, SET>(q, b, n1)) {
      const int i1 = in_img<A, SET>(q, b, n1);
      v = img[irow + i1];
      if (a.conj_in) v = f2conj(v);
      if (sm) {
        float2 s = sm[irow + i1];
        if (a.conj_in) s = f2conj(s);
        v = f2mul(v, s);
      }
      v = f2scale(v, a.dec[1] ? f0 * a.dec[1][i1] : f0);
      if (conj) v = f2conj(v);
    }
    x[q] = v;
  }
  twv.store(s_tw);
  __syncthreads();  // twiddle table
  dft_first<A, SET == kHalf>(x);
  float2* row = s_x + l * (A * 17);
#pragma unroll
  for (int k1 = 0; k1 < A; ++k1) row[k1 * 17 + b] = f2mul(first_out<A>(x, k1), s_tw[k1 * 16 + b]);
  __syncthreads();
  if (!valid) return;
  float2* out = a.fine + (int64_t)c * g.G + (int64_t)img_to_fine(ix, n0, g.nf[0]) * (16 * A);
#pragma unroll
  for (int h = 0; h < (A + 15) / 16; ++h) {
    const int k1 = b + 16 * h;
    if (A % 16 && k1 >= A) break;
    float2 w[16];
#pragma unroll
    for (int q = 0; q < 16; ++q) w[q] = row[k1 * 17 + q];
    dft16(w);
#pragma unroll
    for (int k2 = 0; k2 < 16; ++k2) {
      const float2 v = w[pos16(k2)];
      out[k1 + A * k2] = conj ? f2conj(v) : v;
    }
  }
}

// ---------------------------------------------------------------- x lines
struct Lines2 {
  float2* data;   // ntr grids of G cells
  int64_t G;
  int nf1;        // x stride
  int n_axis;     // image size along x
  int conj;
  unsigned* fmax;  // null, or the largest |re|, |im| written for each transform
  const float2* tw;
};

// blockIdx.x: 16 consecutive y columns; blockIdx.y: transform.  IN / OUT:
// the x entries read / written.
// SQUARE: nf1 = 16 A, the stride as a constant (512^2, 64 transforms: 35 against 44 us)
template <int A, int IN, int OUT, bool SQUARE>
__global__ void __launch_bounds__(kT, kCtas<A>) f2_x_kernel(Lines2 a) {
  const int xs = SQUARE ? 16 * A : a.nf1;
  extern __shared__ float2 s_dyn[];
  float2* const s_tw = s_dyn;
  float2* const s_x = s_tw + 16 * A;
  const TwRegs<A> twv(a.tw);
  const int l = threadIdx.x & 15, b = threadIdx.x >> 4;
  float2* base = a.data + (int64_t)blockIdx.y * a.G + blockIdx.x * kL + l;
  float2 x[A];
#pragma unroll
  for (int q = 0; q < A; ++q) {
    float2 v = make_float2(0.f, 0.f);
    if (in_on<A, IN>(q, b, a.n_axis)) {
      v = base[(16 * q + b) * xs];
      if (a.conj) v = f2conj(v);
    }
    x[q] = v;
  }
  twv.store(s_tw);
  __syncthreads();  // twiddle table
  dft_first<A, IN == kHalf>(x);
#pragma unroll
  for (int k1 = 0; k1 < A; ++k1) s_x[(k1 * 16 + b) * kL + l] = f2mul(first_out<A>(x, k1), s_tw[k1 * 16 + b]);
  __syncthreads();
  float mx = 0.f;
#pragma unroll
  for (int h = 0; h < (A + 15) / 16; ++h) {
    const int k1 = b + 16 * h;
    if (A % 16 && k1 >= A) break;
    float2 w[16];
#pragma unroll
    for (int q = 0; q < 16; ++q) w[q] = s_x[(k1 * 16 + q) * kL + l];
    dft16<false, OUT == kHalf>(w);
#pragma unroll
    for (int k2 = 0; k2 < 16; ++k2) {
      if (out_on<A, OUT>(k1, k2, a.n_axis)) {
        const float2 v = w[pos16(k2)];
        base[(k1 + A * k2) * xs] = a.conj ? f2conj(v) : v;
        if (OUT == kAll) mx = fmaxf(mx, fmaxf(fabsf(v.x), fabsf(v.y)));
      }
    }
  }
  if (OUT == kAll && a.fmax) {
    // the atomic only where this warp raises the maximum
    const unsigned m = __reduce_max_sync(0xffffffffu, __float_as_uint(mx));
    unsigned* const p = a.fmax + blockIdx.y;
    if ((threadIdx.x & 31) == 0 && m > *reinterpret_cast<volatile unsigned*>(p)) atomicMax(p, m);
  }
}

// ---------------------------------------------------------------- y lines, crop fused
// blockIdx.x: 16 consecutive x image rows; blockIdx.y: transform.  SET: the y modes.
// ORDERED, conj(s_c) v_c takes the place of the row's first n1 cells, which this CTA
// alone reads, before its first store (one coil: the image).
template <int A, int SET, bool ORDERED>
__global__ void __launch_bounds__(kT, kCtas<A>)
f2_crop_y_kernel(CropArgs a, float2* fine, const float2* __restrict__ tw, int conj) {
  extern __shared__ float2 s_dyn[];
  float2* const s_tw = s_dyn;
  float2* const s_x = s_tw + 16 * A;
  const Geom& g = a.g;
  const int n0 = g.n[0], n1 = g.n[1];
  const TwRegs<A> twv(tw);
  const int b = threadIdx.x & 15, l = threadIdx.x >> 4;
  const int ix = blockIdx.x * kL + l;
  const bool valid = ix < n0;
  const int c = blockIdx.y;
  const int64_t frow = (int64_t)c * g.G + (int64_t)img_to_fine(valid ? ix : 0, n0, g.nf[0]) * (16 * A);
  const float2* in = a.fine + frow;
  float2 x[A];
#pragma unroll
  for (int q = 0; q < A; ++q) {
    const float2 v = valid ? in[16 * q + b] : make_float2(0.f, 0.f);
    x[q] = conj ? f2conj(v) : v;
  }
  twv.store(s_tw);
  __syncthreads();  // twiddle table
  dft_first<A>(x);
  float2* row = s_x + l * (A * 17);
#pragma unroll
  for (int k1 = 0; k1 < A; ++k1) row[k1 * 17 + b] = f2mul(first_out<A>(x, k1), s_tw[k1 * 16 + b]);
  __syncthreads();
  if (!valid) return;
  float f0 = a.scale;
  if (a.dec[0]) f0 *= a.dec[0][ix];
  const int64_t irow = (int64_t)ix * n1;
#pragma unroll
  for (int h = 0; h < (A + 15) / 16; ++h) {
    const int k1 = b + 16 * h;
    if (A % 16 && k1 >= A) break;
    float2 w[16];
#pragma unroll
    for (int q = 0; q < 16; ++q) w[q] = row[k1 * 17 + q];
    dft16<false, SET == kHalf>(w);
#pragma unroll
    for (int k2 = 0; k2 < 16; ++k2) {
      if (!out_on<A, SET>(k1, k2, n1)) continue;
      const int i1 = mode_to_img(k1 + A * k2, n1, 16 * A);
      float2 v = w[pos16(k2)];
      if (conj) v = f2conj(v);
      v = f2scale(v, a.dec[1] ? f0 * a.dec[1][i1] : f0);
      if (a.smaps) {
        const float2 s = a.smaps[(int64_t)c * g.Nimg + irow + i1];
        const float2 p = make_float2(s.x * v.x + s.y * v.y, s.x * v.y - s.y * v.x);
        if constexpr (!ORDERED) {
          atomicAdd(a.out + irow + i1, p);
        } else if (a.ntr > 1) {
          fine[frow + i1] = p;
        } else {
          float2* dst = a.out + irow + i1;
          *dst = a.accumulate ? f2add(p, *dst) : p;
        }
      } else {
        float2* dst = a.out + (int64_t)c * g.Nimg + irow + i1;
        if (a.accumulate) v = f2add(v, *dst);
        *dst = v;
      }
    }
  }
}

// The coils' products of an ordered pass, summed as the crop pass of the other grids
// does.  blockIdx.x: 256 pixels of the image row blockIdx.y.  Bound by the read of what
// the crop has just left in L2.  The Toeplitz Gram, which has no other atomics, takes
// it: 384^2 images (768^2 cells), 16 coils 155 -> 157 us, 40 415 -> 428 against atomics.
// The adjoint's spreading adds with atomics anyway; 480 effective coils of 256^2 images
// in passes of 64 4.65 against 4.73 ms for op + adj.
__global__ void __launch_bounds__(kT) f2_coil_sum_kernel(CropArgs a, const float2* __restrict__ fine) {
  const Geom& g = a.g;
  const int i1 = blockIdx.x * kT + threadIdx.x, ix = blockIdx.y;
  if (i1 >= g.n[1]) return;
  const float2* p = fine + (int64_t)img_to_fine(ix, g.n[0], g.nf[0]) * g.nf[1] + i1;
  float2 s = make_float2(0.f, 0.f);
#pragma unroll 8
  for (int c = 0; c < a.ntr; ++c) s = f2add(s, p[(int64_t)c * g.G]);
  float2* const dst = a.out + (int64_t)ix * g.n[1] + i1;
  if (a.accumulate) s = f2add(s, *dst);
  *dst = s;
}

// ---------------------------------------------------------------- x lines of the Toeplitz Gram
// 512-point x axis.  Forward x transform (x-mode entries in), multiply by the real spectrum K,
// inverse x transform (x-mode entries out), per (y column, transform).
// blockIdx.x: 16 consecutive y columns; blockIdx.y: transform
template <int SET, bool SQUARE>
__global__ void __launch_bounds__(kT, 2)
f2_x_kmul_kernel(float2* data, int64_t G, int nf1, int n0, const float* __restrict__ K,
                   const float2* __restrict__ tw) {
  const int kN = SQUARE ? 512 : nf1;  // x stride
  extern __shared__ float2 s_dyn[];
  float2* const s_tw = s_dyn;
  float2* const s_x = s_tw + 512;
  const TwRegs<32> twv(tw);
  const int l = threadIdx.x & 15, b = threadIdx.x >> 4;
  const int y = blockIdx.x * kL + l;
  float2* base = data + (int64_t)blockIdx.y * G + y;
  float2 x[32];
#pragma unroll
  for (int q = 0; q < 32; ++q)
    x[q] = in_on<32, SET>(q, b, n0) ? base[(16 * q + b) * kN] : make_float2(0.f, 0.f);
  twv.store(s_tw);
  __syncthreads();  // twiddle table
  dft32<SET == kHalf>(x);
#pragma unroll
  for (int k1 = 0; k1 < 32; ++k1) s_x[(k1 * 16 + b) * kL + l] = f2mul(x[k1], s_tw[k1 * 16 + b]);
  __syncthreads();
  // X[b + 16 h + 32 k2] -> conj(K X) as the inverse transform's x[16 (h + 2 k2) + b]
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int k1 = b + 16 * h;
    float2 w[16];
#pragma unroll
    for (int q = 0; q < 16; ++q) w[q] = s_x[(k1 * 16 + q) * kL + l];
    dft16(w);
#pragma unroll
    for (int k2 = 0; k2 < 16; ++k2)
      x[h + 2 * k2] = f2conj(f2scale(w[pos16(k2)], K[(k1 + 32 * k2) * kN + y]));
  }
  dft32(x);
  __syncthreads();  // every thread has read its forward exchange entries
#pragma unroll
  for (int k1 = 0; k1 < 32; ++k1) s_x[(k1 * 16 + b) * kL + l] = f2mul(x[k1], s_tw[k1 * 16 + b]);
  __syncthreads();
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int k1 = b + 16 * h;
    float2 w[16];
#pragma unroll
    for (int q = 0; q < 16; ++q) w[q] = s_x[(k1 * 16 + q) * kL + l];
    dft16<false, SET == kHalf>(w);
#pragma unroll
    for (int k2 = 0; k2 < 16; ++k2)
      if (out_on<32, SET>(k1, k2, n0)) base[(k1 + 32 * k2) * kN] = f2conj(w[pos16(k2)]);
  }
}

template <typename F>
cudaError_t set_smem(F* k, size_t bytes) {
  return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

template <int A>
cudaError_t prepare_a() {
  cudaError_t e = cudaSuccess;
  auto chk = [&](cudaError_t r) {
    if (e == cudaSuccess) e = r;
  };
  chk(set_smem(f2_pad_y_kernel<A, kHalf>, y_smem<A>()));
  chk(set_smem(f2_pad_y_kernel<A, kModes>, y_smem<A>()));
  chk(set_smem(f2_crop_y_kernel<A, kHalf, false>, y_smem<A>()));
  chk(set_smem(f2_crop_y_kernel<A, kHalf, true>, y_smem<A>()));
  chk(set_smem(f2_crop_y_kernel<A, kModes, false>, y_smem<A>()));
  chk(set_smem(f2_crop_y_kernel<A, kModes, true>, y_smem<A>()));
  chk(set_smem(f2_x_kernel<A, kHalf, kAll, true>, x_smem<A>()));
  chk(set_smem(f2_x_kernel<A, kModes, kAll, true>, x_smem<A>()));
  chk(set_smem(f2_x_kernel<A, kAll, kHalf, true>, x_smem<A>()));
  chk(set_smem(f2_x_kernel<A, kAll, kModes, true>, x_smem<A>()));
  chk(set_smem(f2_x_kernel<A, kModes, kAll, false>, x_smem<A>()));
  chk(set_smem(f2_x_kernel<A, kAll, kModes, false>, x_smem<A>()));
  return e;
}

template <int A>
void pad_y_a(const PadArgs& pa, const float2* tw, int conj, cudaStream_t st) {
  const dim3 gy((pa.g.n[0] + kL - 1) / kL, pa.ntr);
  if (pa.g.n[1] == 8 * A) f2_pad_y_kernel<A, kHalf><<<gy, kT, y_smem<A>(), st>>>(pa, tw, conj);
  else f2_pad_y_kernel<A, kModes><<<gy, kT, y_smem<A>(), st>>>(pa, tw, conj);
}
template <int A>
void crop_y_a(const CropArgs& ca, float2* fine, const float2* tw, int conj, cudaStream_t st) {
  const dim3 gy((ca.g.n[0] + kL - 1) / kL, ca.ntr);
  const bool half = ca.g.n[1] == 8 * A, ordered = ca.smaps && (ca.ordered || ca.ntr == 1);
  auto k = half ? (ordered ? f2_crop_y_kernel<A, kHalf, true> : f2_crop_y_kernel<A, kHalf, false>)
                : (ordered ? f2_crop_y_kernel<A, kModes, true> : f2_crop_y_kernel<A, kModes, false>);
  k<<<gy, kT, y_smem<A>(), st>>>(ca, fine, tw, conj);
}
template <int A>
void x_lines_a(const Lines2& x, int ntr, bool in_prune, cudaStream_t st) {
  const dim3 gx(x.nf1 / kL, ntr);
  const bool half = x.n_axis == 8 * A;
  const bool square = x.nf1 == 16 * A;
  auto k = in_prune ? (!square ? f2_x_kernel<A, kModes, kAll, false>
                       : half  ? f2_x_kernel<A, kHalf, kAll, true>
                               : f2_x_kernel<A, kModes, kAll, true>)
                    : (!square ? f2_x_kernel<A, kAll, kModes, false>
                       : half  ? f2_x_kernel<A, kAll, kHalf, true>
                               : f2_x_kernel<A, kAll, kModes, true>);
  k<<<gx, kT, x_smem<A>(), st>>>(x);
}

// calls f with the axis length nf / 16 as a compile-time constant
template <typename F>
void with_axis(int nf, F&& f) {
  switch (nf) {
    case 256: return f(std::integral_constant<int, 16>{});
    case 384: return f(std::integral_constant<int, 24>{});
    case 512: return f(std::integral_constant<int, 32>{});
    case 640: return f(std::integral_constant<int, 40>{});
    default: return f(std::integral_constant<int, 48>{});
  }
}

void pad_y(const PadArgs& pa, const Twiddles& tw, int conj, cudaStream_t st) {
  with_axis(pa.g.nf[1], [&](auto A) { pad_y_a<decltype(A)::value>(pa, tw.t[1], conj, st); });
}
cudaError_t crop_y(const CropArgs& ca, float2* fine, const Twiddles& tw, int conj, cudaStream_t st) {
  const bool sum = ca.smaps && ca.ntr > 1;
  if (sum && !ca.ordered && !ca.accumulate) {
    cudaError_t e = cudaMemsetAsync(ca.out, 0, sizeof(float2) * (size_t)ca.g.Nimg, st);
    if (e != cudaSuccess) return e;
  }
  with_axis(ca.g.nf[1], [&](auto A) { crop_y_a<decltype(A)::value>(ca, fine, tw.t[1], conj, st); });
  if (sum && ca.ordered)
    f2_coil_sum_kernel<<<dim3((ca.g.n[1] + kT - 1) / kT, ca.g.n[0]), kT, 0, st>>>(ca, fine);
  return cudaGetLastError();
}
void x_lines(float2* fine, const Geom& g, const Twiddles& tw, int ntr, bool in_prune, int conj, unsigned* fmax,
             cudaStream_t st) {
  Lines2 x{};
  x.data = fine;
  x.G = g.G;
  x.nf1 = g.nf[1];
  x.n_axis = g.n[0];
  x.conj = conj;
  x.fmax = fmax;
  x.tw = tw.t[0];
  with_axis(g.nf[0], [&](auto A) { x_lines_a<decltype(A)::value>(x, ntr, in_prune, st); });
}

}  // namespace

bool fft2d_fits(const Geom& g) {
  if (g.dim != 2) return false;
  for (int d = 0; d < 2; ++d)
    if (g.nf[d] % 128 || g.nf[d] < 256 || g.nf[d] > 768) return false;
  return true;
}

cudaError_t fft2d_prepare(const Geom& g) {
  cudaError_t e = cudaSuccess;
  for (int d = 0; d < 2; ++d)
    with_axis(g.nf[d], [&](auto A) {
      if (e == cudaSuccess) e = prepare_a<decltype(A)::value>();
    });
  for (auto k : {f2_x_kmul_kernel<kHalf, true>, f2_x_kmul_kernel<kModes, true>, f2_x_kmul_kernel<kModes, false>})
    if (e == cudaSuccess) e = set_smem(k, x_smem<32>());
  return e;
}

cudaError_t launch_fft2d_op(const PadArgs& pa, const Twiddles& tw, int isign, cudaStream_t st) {
  const int conj = isign > 0;
  pad_y(pa, tw, conj, st);
  x_lines(pa.fine, pa.g, tw, pa.ntr, true, conj, pa.fmax, st);
  return cudaGetLastError();
}

cudaError_t launch_fft2d_adj(const CropArgs& ca, float2* fine, const Twiddles& tw, int isign,
                             cudaStream_t st) {
  const int conj = isign > 0;
  x_lines(fine, ca.g, tw, ca.ntr, false, conj, nullptr, st);
  return crop_y(ca, fine, tw, conj, st);
}

cudaError_t launch_fft2d_gram(const PadArgs& pa, const CropArgs& ca, const float* K,
                              const Twiddles& tw, cudaStream_t st) {
  const Geom& g = pa.g;
  if (g.nf[0] != 512) return cudaErrorInvalidValue;
  pad_y(pa, tw, 0, st);
  const dim3 gx(g.nf[1] / kL, pa.ntr);
  auto k = g.nf[1] != 512 ? f2_x_kmul_kernel<kModes, false>
           : g.n[0] == 256 ? f2_x_kmul_kernel<kHalf, true>
                           : f2_x_kmul_kernel<kModes, true>;
  k<<<gx, kT, x_smem<32>(), st>>>(pa.fine, g.G, g.nf[1], g.n[0], K, tw.t[0]);
  return crop_y(ca, pa.fine, tw, 1, st);
}

}  // namespace gbn
