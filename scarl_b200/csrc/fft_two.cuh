// fft_two.cuh -- line transforms in two in-register stages (the "four-step"
// factorisation): N = A B, A and B <= 32.  With k = t + B r and n = m + A s
// (t, s < B; r, m < A),
//   Y[t][m] = sum_r x[t + B r] e^{+2 pi i m r / A}      DFT-A, one a work item t
//   Y'      = Y e^{+2 pi i m t / N}
//   y[m + A s] = sum_t Y'[t][m] e^{+2 pi i s t / B}     DFT-B, one a work item m
// One hand-off through shared memory and one twiddle a value, where radix
// stages of at most 16 take two to four of each.
#pragma once

#include "fft_engine.cuh"

namespace scarl {

// ---------------------------------------------------------------------------
// Compile-time unit roots: cos and sin of 2 pi j / n in double, from Taylor
// series on |x| <= pi/4 after an exact integer reduction to the first octant.
// ---------------------------------------------------------------------------
__host__ __device__ constexpr double cx_sin_oct(double x) {
  double term = x, sum = x;
  for (int i = 1; i < 14; ++i) {
    term *= -x * x / (double)((2 * i) * (2 * i + 1));
    sum += term;
  }
  return sum;
}
__host__ __device__ constexpr double cx_cos_oct(double x) {
  double term = 1.0, sum = 1.0;
  for (int i = 1; i < 14; ++i) {
    term *= -x * x / (double)((2 * i - 1) * (2 * i));
    sum += term;
  }
  return sum;
}
// (cos, sin)(2 pi j / n): quadrant q = floor(4 j / n), remainder angle
// r = 2 pi num / (4 n) with num = 4 j - q n in [0, n); r > pi / 4 uses the
// complement 2 pi (n - num) / (4 n).
__host__ __device__ constexpr void cx_root(long long j, long long n, double& c, double& s) {
  constexpr double kTwoPi = 6.283185307179586476925286766559;
  j %= n;
  if (j < 0) j += n;
  const long long q = (4 * j) / n, num = 4 * j - q * n;
  double c0 = 0.0, s0 = 0.0;
  if (2 * num <= n) {
    const double x = kTwoPi * (double)num / (double)(4 * n);
    c0 = cx_cos_oct(x);
    s0 = cx_sin_oct(x);
  } else {
    const double x = kTwoPi * (double)(n - num) / (double)(4 * n);
    c0 = cx_sin_oct(x);
    s0 = cx_cos_oct(x);
  }
  if (q == 0) { c = c0; s = s0; }
  else if (q == 1) { c = -s0; s = c0; }
  else if (q == 2) { c = -c0; s = -s0; }
  else { c = s0; s = -c0; }
}

template <int N> struct RootTable {
  double c[N], s[N];
  constexpr RootTable() : c(), s() {
    for (int j = 0; j < N; ++j) {
      double cc = 0.0, ss = 0.0;
      cx_root(j, N, cc, ss);
      c[j] = cc;
      s[j] = ss;
    }
  }
};
template <int N> __device__ constexpr RootTable<N> kRootTable = RootTable<N>();

// ---------------------------------------------------------------------------
// In-register inverse DFT of N2 = P Q points (P a power of two <= 32, Q = 1,
// 3, 5 or 7), natural order in and out: with k = q + Q p and n = np + P nq,
// DFT-P over p for each q, twiddle e^{+2 pi i np q / N2}, DFT-Q over q.
// ---------------------------------------------------------------------------
template <int N2, typename C> __device__ __forceinline__ void dft_natural(C* v) {
  using T = decltype(v[0].x);
  constexpr int Q = odd_part(N2), P = N2 / Q;
  static_assert(P <= 32 && (Q == 1 || Q == 3 || Q == 5 || Q == 7), "in-register length");
  if constexpr (Q == 1) {
    dft_reg<P>(v);
    C t[P];
#pragma unroll
    for (int i = 0; i < P; ++i) t[i] = v[operm<P>(i)];
#pragma unroll
    for (int i = 0; i < P; ++i) v[i] = t[i];
  } else if constexpr (P == 1) {
    dft_odd<Q>(v);
  } else {
    C y[N2];  // y[q P + np]
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      C t[P];
#pragma unroll
      for (int p = 0; p < P; ++p) t[p] = v[q + Q * p];
      dft_reg<P>(t);
#pragma unroll
      for (int np = 0; np < P; ++np) y[q * P + np] = t[operm<P>(np)];
    }
#pragma unroll
    for (int q = 1; q < Q; ++q)
#pragma unroll
      for (int np = 1; np < P; ++np) {
        const int j = (np * q) % N2;
        const T c = (T)kRootTable<N2>.c[j], s = (T)kRootTable<N2>.s[j];
        const C d = y[q * P + np];
        y[q * P + np] = mk(d.x * c - d.y * s, d.x * s + d.y * c);
      }
#pragma unroll
    for (int np = 0; np < P; ++np) {
      C t[Q];
#pragma unroll
      for (int q = 0; q < Q; ++q) t[q] = y[q * P + np];
      dft_odd<Q>(t);
#pragma unroll
      for (int nq = 0; nq < Q; ++nq) v[np + P * nq] = t[nq];
    }
  }
}

}  // namespace scarl
