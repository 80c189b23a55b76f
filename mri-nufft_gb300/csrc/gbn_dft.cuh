// Complex helpers and in-register DFTs of 2 to 48 points shared by the fused
// line transforms (gbn_fft3d.cu, gbn_fft2d.cu).  Exponent sign -1
// throughout; a +1 transform conjugates its inputs and outputs.
#pragma once

#include <cuda_runtime.h>

namespace gbn {
namespace dft {

__device__ __forceinline__ float2 f2add(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 f2sub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 f2mul(float2 a, float2 b) {
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ float2 f2conj(float2 a) { return make_float2(a.x, -a.y); }
__device__ __forceinline__ float2 f2scale(float2 a, float s) { return make_float2(a.x * s, a.y * s); }

// 4-point DFT, exponent sign -1, in place
__device__ __forceinline__ void dft4(float2& a0, float2& a1, float2& a2, float2& a3) {
  const float2 t0 = f2add(a0, a2), t1 = f2sub(a0, a2), t2 = f2add(a1, a3), t3 = f2sub(a1, a3);
  a0 = f2add(t0, t2);
  a2 = f2sub(t0, t2);
  a1 = make_float2(t1.x + t3.y, t1.y - t3.x);  // t1 - i t3
  a3 = make_float2(t1.x - t3.y, t1.y + t3.x);  // t1 + i t3
}

// 4-point DFT whose inputs a1, a2 are zero (not read)
__device__ __forceinline__ void dft4_in03(float2& a0, float2& a1, float2& a2, float2& a3) {
  const float2 p = a0, q = a3;
  a0 = f2add(p, q);
  a2 = f2sub(p, q);
  a1 = make_float2(p.x - q.y, p.y + q.x);  // p + i q
  a3 = make_float2(p.x + q.y, p.y - q.x);  // p - i q
}

// 4-point DFT of which only the outputs a0, a3 are used (a1, a2 are left stale)
__device__ __forceinline__ void dft4_out03(float2& a0, float2& a1, float2& a2, float2& a3) {
  const float2 t0 = f2add(a0, a2), t1 = f2sub(a0, a2), t2 = f2add(a1, a3), t3 = f2sub(a1, a3);
  a0 = f2add(t0, t2);
  a3 = make_float2(t1.x - t3.y, t1.y + t3.x);
}

// 16-point DFT, exponent sign -1: x[n] in natural order in, X[k] at x[pos16(k)] out.
// HALF_IN: x[4 .. 11] are zero and not read (the inputs of a 128-mode axis,
// n = 16 q + b with q < 4 or q >= 12); HALF_OUT: only X[k], k < 4 or k >= 12,
// are computed (the outputs such an axis keeps).  The IEEE arithmetic does
// not let the compiler drop additions of constant zeros by itself.
__device__ __forceinline__ int pos16(int k) { return 4 * (k & 3) + (k >> 2); }

template <bool HALF_IN = false, bool HALF_OUT = false>
__device__ __forceinline__ void dft16(float2 (&x)[16]) {
  // W16^k = (cos(2 pi k / 16), -sin(2 pi k / 16))
  constexpr float c1 = 0.92387953251128674f;  // cos(pi / 8)
  constexpr float s1 = 0.38268343236508977f;  // sin(pi / 8)
  constexpr float r2 = 0.70710678118654752f;  // sqrt(1 / 2)
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    if (HALF_IN) dft4_in03(x[r], x[r + 4], x[r + 8], x[r + 12]);
    else dft4(x[r], x[r + 4], x[r + 8], x[r + 12]);
  }
  // x[r + 4 s] *= W16^(r s)
  x[5] = f2mul(x[5], make_float2(c1, -s1));    // r 1, s 1
  x[9] = f2mul(x[9], make_float2(r2, -r2));    // r 1, s 2
  x[13] = f2mul(x[13], make_float2(s1, -c1));  // r 1, s 3
  x[6] = f2mul(x[6], make_float2(r2, -r2));    // r 2, s 1
  x[10] = make_float2(x[10].y, -x[10].x);      // r 2, s 2: W16^4 = -i
  x[14] = f2mul(x[14], make_float2(-r2, -r2)); // r 2, s 3: W16^6
  x[7] = f2mul(x[7], make_float2(s1, -c1));    // r 3, s 1: W16^3
  x[11] = f2mul(x[11], make_float2(-r2, -r2)); // r 3, s 2: W16^6
  x[15] = f2mul(x[15], make_float2(-c1, s1));  // r 3, s 3: W16^9
#pragma unroll
  for (int s = 0; s < 4; ++s) {
    if (HALF_OUT) dft4_out03(x[4 * s], x[4 * s + 1], x[4 * s + 2], x[4 * s + 3]);
    else dft4(x[4 * s], x[4 * s + 1], x[4 * s + 2], x[4 * s + 3]);
  }
}

// cos and sin of 2 pi k / N in double precision at compile time (power series on
// the first octant's angle)
constexpr double series_cos(double x) {
  double t = 1.0, s = 1.0;
  for (int i = 1; i < 12; ++i) {
    t *= -x * x / ((2 * i - 1) * (2 * i));
    s += t;
  }
  return s;
}
constexpr double series_sin(double x) {
  double t = x, s = x;
  for (int i = 1; i < 12; ++i) {
    t *= -x * x / ((2 * i) * (2 * i + 1));
    s += t;
  }
  return s;
}
// W_N^k = (cos(2 pi k / N), -sin(2 pi k / N)), 0 <= 8 k <= N
template <int N>
struct Octant {
  float c[N / 8 + 1] = {}, s[N / 8 + 1] = {};
  constexpr Octant() {
    for (int k = 0; k <= N / 8; ++k) {
      const double a = 2.0 * 3.14159265358979323846 * k / N;
      c[k] = (float)series_cos(a);
      s[k] = (float)series_sin(a);
    }
  }
};
// v * W_N^k; k is a constant after unrolling.  N a multiple of 8 up to symmetry:
// other N are taken on the finer grid of 8 N.
template <int N>
__device__ __forceinline__ float2 mul_root(float2 v, int k) {
  constexpr int M = 8 * N;
  constexpr Octant<M> oct{};
  int e = 8 * k % M;          // in units of 1 / M turn
  const int q = e / (M / 4);  // quarter turns
  e -= q * (M / 4);
  if (e != 0) {
    const bool hi = e > M / 8;
    const int f = hi ? M / 4 - e : e;
    const float c = hi ? oct.s[f] : oct.c[f], s = hi ? oct.c[f] : oct.s[f];
    v = f2mul(v, make_float2(c, -s));
  }
  switch (q) {  // (-i)^q
    case 0: return v;
    case 1: return make_float2(v.y, -v.x);
    case 2: return make_float2(-v.x, -v.y);
    default: return make_float2(-v.y, v.x);
  }
}

__device__ __forceinline__ void dft3(float2& a0, float2& a1, float2& a2) {
  constexpr float h = 0.86602540378443865f;  // sin(2 pi / 3)
  const float2 t = f2add(a1, a2), d = f2scale(f2sub(a1, a2), h);
  const float2 m = make_float2(a0.x - 0.5f * t.x, a0.y - 0.5f * t.y);
  a0 = f2add(a0, t);
  a1 = make_float2(m.x + d.y, m.y - d.x);  // m - i d
  a2 = make_float2(m.x - d.y, m.y + d.x);
}
__device__ __forceinline__ void dft5(float2& a0, float2& a1, float2& a2, float2& a3, float2& a4) {
  constexpr float c1 = 0.30901699437494742f, c2 = -0.80901699437494742f;  // cos(2 pi / 5), cos(4 pi / 5)
  constexpr float s1 = 0.95105651629515357f, s2 = 0.58778525229247313f;   // sin(2 pi / 5), sin(4 pi / 5)
  const float2 p = f2add(a1, a4), q = f2add(a2, a3), u = f2sub(a1, a4), v = f2sub(a2, a3);
  const float2 m1 = make_float2(a0.x + c1 * p.x + c2 * q.x, a0.y + c1 * p.y + c2 * q.y);
  const float2 m2 = make_float2(a0.x + c2 * p.x + c1 * q.x, a0.y + c2 * p.y + c1 * q.y);
  const float2 n1 = make_float2(s1 * u.x + s2 * v.x, s1 * u.y + s2 * v.y);
  const float2 n2 = make_float2(s2 * u.x - s1 * v.x, s2 * u.y - s1 * v.y);
  a0 = make_float2(a0.x + p.x + q.x, a0.y + p.y + q.y);
  a1 = make_float2(m1.x + n1.y, m1.y - n1.x);  // m1 - i n1
  a4 = make_float2(m1.x - n1.y, m1.y + n1.x);
  a2 = make_float2(m2.x + n2.y, m2.y - n2.x);
  a3 = make_float2(m2.x - n2.y, m2.y + n2.x);
}

// N-point DFT, natural order in, N = 2^a 3^b 5^c with small factors: radix 4 (or
// 2) steps down to 2, 3, 4 or 5 points.  HALF_IN (N a multiple of 4): the middle
// half of the inputs is zero and not read.  Outputs that the caller does not use
// cost nothing.  Natural order out with NAT, else X[k] at x[dftn_pos<N>(k)]: the
// copies of the natural order are free, but kept the compiler from overlapping
// the loads of the 3D passes that follow (pad 45 against 56 us).
template <int N>
__host__ __device__ constexpr int dftn_pos(int k) {
  return N % 4 ? k : (N / 4) * (k & 3) + (k >> 2);
}
template <int N, bool HALF_IN = false, bool NAT = true>
__device__ __forceinline__ void dftn(float2 (&x)[N]) {
  if constexpr (N == 2) {
    const float2 t = x[0];
    x[0] = f2add(t, x[1]);
    x[1] = f2sub(t, x[1]);
  } else if constexpr (N == 3) {
    dft3(x[0], x[1], x[2]);
  } else if constexpr (N == 4) {
    dft4(x[0], x[1], x[2], x[3]);
  } else if constexpr (N == 5) {
    dft5(x[0], x[1], x[2], x[3], x[4]);
  } else if constexpr (N == 16) {
    dft16<HALF_IN>(x);
    if (!NAT) return;
    float2 y[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) y[k] = x[pos16(k)];
#pragma unroll
    for (int k = 0; k < 16; ++k) x[k] = y[k];
  } else {
    constexpr int P = N % 4 == 0 ? 4 : 2, Q = N / P;
    static_assert(P * Q == N && (!HALF_IN || P == 4), "unsupported DFT length");
    // n = Q a + b, k = k1 + P k2
    float2 t[P][Q];
#pragma unroll
    for (int b = 0; b < Q; ++b) {
      if constexpr (P == 4) {
        float2 v0 = x[b], v1 = x[Q + b], v2 = x[2 * Q + b], v3 = x[3 * Q + b];
        if (HALF_IN) dft4_in03(v0, v1, v2, v3);
        else dft4(v0, v1, v2, v3);
        t[0][b] = v0;
        t[1][b] = mul_root<N>(v1, b);
        t[2][b] = mul_root<N>(v2, 2 * b);
        t[3][b] = mul_root<N>(v3, 3 * b);
      } else {
        t[0][b] = f2add(x[b], x[Q + b]);
        t[1][b] = mul_root<N>(f2sub(x[b], x[Q + b]), b);
      }
    }
#pragma unroll
    for (int k1 = 0; k1 < P; ++k1) {
      dftn<Q>(t[k1]);
#pragma unroll
      for (int k2 = 0; k2 < Q; ++k2) x[NAT ? k1 + P * k2 : Q * k1 + k2] = t[k1][k2];
    }
  }
}

}  // namespace dft
}  // namespace gbn
