// gen_two.cuh -- passes 1 and 2 of the padded generator (synthesis + inverse
// DFT along z; inverse DFT along y) with each line in two in-register stages
// (fft_two.cuh).  LB consecutive kx a block, lanes across them; a line has T =
// B threads, one DFT-A each in stage 1, and ceil(A / B) rounds of DFT-B in
// stage 2.  One hand-off through shared memory: pass 1 synthesises into the
// same area (each thread its own modes), pass 2 reads its columns straight from
// global memory, A loads in flight a thread.
#pragma once

#include "fft_two.cuh"
#include "gen_kernels.cuh"

namespace scarl {

// Factors of a line of N values (A even: kz and kz + N/2, the two modes of one
// draw, then fall to one thread).
template <typename T, int N> struct ColLen {
  static constexpr int A = N == 32 ? 8 : N == 48 ? 6 : N == 64 ? 8 : N == 80 ? 10 : N == 96 ? 12 : N == 112 ? 14
                         : N == 128 ? 16 : N == 160 ? 10 : N == 192 ? 12 : N == 224 ? 14 : N == 256 ? 16
                         : N == 320 ? 20 : N == 384 ? 24 : N == 448 ? 28 : N == 512 ? 16 : N == 640 ? 20
                         : N == 768 ? 24 : N == 896 ? 28 : N == 1024 ? 32 : 1;
  static constexpr int B = N / A;
  static constexpr int MAXR = sizeof(T) == 4 ? 32 : 16;
  static constexpr bool valid() { return A > 1 && A * B == N && A % 2 == 0 && A <= MAXR && B <= MAXR; }
};
template <typename T, int N> struct ColCfg {
  using Len = ColLen<T, N>;
  static constexpr int A = Len::A, B = Len::B, LB = sizeof(T) == 4 ? 8 : 4;  // 64-byte runs of kx
  static constexpr int THREADS = LB * B, ROUNDS = (A + B - 1) / B;
  static constexpr int XROW = B % 2 == 0 ? B + 1 : B;  // rows an odd number of 64-byte runs apart
  static constexpr int SMEM = (A * XROW > N ? A * XROW : N) * LB * 2 * (int)sizeof(T);
  // resident blocks asked of the compiler: about 2 R + 32 registers a thread
  // (R: the longer in-register DFT) in FP32, twice the values in FP64 (448: 35
  // -> 27 us in pass 2); DFT-32 needs what it takes (capped, 640 points went
  // from 113 to 129 us in pass 1)
  static constexpr int R = A > B ? A : B;
  static constexpr int REGS = sizeof(T) == 4 ? 2 * R + 32 : 4 * R + 40;
  static constexpr int FIT = 65536 / (REGS * THREADS);
  static constexpr int MINB = R >= 32 || FIT < 1 ? 1 : FIT > 32 ? 32 : FIT;
  static constexpr bool valid() { return Len::valid() && THREADS <= 1024 && SMEM <= 200 * 1024; }
};

// Twiddle, hand-off and stage 2 of a line whose stage-1 outputs sit in v:
// store(n, y_n) takes the outputs n = m + A s.
template <typename T, int N, class Store>
__device__ __forceinline__ void col_finish(cplx_t<T>* sm, cplx_t<T>* v, int b, int t, const cplx_t<T>* __restrict__ tw,
                                           Store&& store) {
  using Cfg = ColCfg<T, N>;
  using C = cplx_t<T>;
  constexpr int A = Cfg::A, B = Cfg::B, LB = Cfg::LB;
#pragma unroll
  for (int m = 1; m < A; ++m) v[m] = cmul(v[m], __ldg(tw + m * t));
#pragma unroll
  for (int m = 0; m < A; ++m) sm[(m * Cfg::XROW + t) * LB + b] = v[m];
  __syncthreads();
#pragma unroll 1
  for (int m = t; m < A; m += B) {
    C u[B];
#pragma unroll
    for (int k = 0; k < B; ++k) u[k] = sm[(m * Cfg::XROW + k) * LB + b];
    dft_natural<B>(u);
#pragma unroll
    for (int s = 0; s < B; ++s) store(m + A * s, u[s]);
  }
}

template <typename T, int N>
__device__ __forceinline__ void gen_z_two_body(const GenArgs& a, int bx, int ky) {
  using Cfg = ColCfg<T, N>;
  using C = cplx_t<T>;
  constexpr int A = Cfg::A, B = Cfg::B, LB = Cfg::LB;
  extern __shared__ __align__(16) unsigned char smraw[];
  C* sm = reinterpret_cast<C*>(smraw);
  const int b = threadIdx.x % LB, t = threadIdx.x / LB;
  const int kx = bx * LB + b;
  const bool valid = kx < a.Hx;
  C v[A];
  if (valid) {
    synth_line<T>(a, kx, ky, [&](int d) { return t + B * d; }, A / 2, N, [&](int kz, C x) { sm[kz * LB + b] = x; });
#pragma unroll
    for (int r = 0; r < A; ++r) v[r] = sm[(t + B * r) * LB + b];
  } else {
#pragma unroll
    for (int r = 0; r < A; ++r) v[r] = mk(T(0), T(0));
  }
  dft_natural<A>(v);
  __syncthreads();  // every thread has read its modes
  const int Nz = a.Nout[2];
  const size_t zstride = (size_t)a.P[1] * a.Hpad;
  C* wcol = static_cast<C*>(a.work) + (size_t)ky * a.Hpad + kx;
  col_finish<T, N>(sm, v, b, t, static_cast<const C*>(a.tw_z), [&](int z, C y) {
    if (valid && z < Nz) wcol[(size_t)z * zstride] = y;
  });
}

template <typename T, int N>
__device__ __forceinline__ void mid_y_two_body(const GenArgs& a, int bx, int z) {
  using Cfg = ColCfg<T, N>;
  using C = cplx_t<T>;
  constexpr int A = Cfg::A, B = Cfg::B, LB = Cfg::LB;
  extern __shared__ __align__(16) unsigned char smraw[];
  C* sm = reinterpret_cast<C*>(smraw);
  const int b = threadIdx.x % LB, t = threadIdx.x / LB;
  const int kx = bx * LB + b;
  const bool valid = kx < a.Hx;
  const size_t pitch = (size_t)a.Hpad;
  C* col = static_cast<C*>(a.work) + (size_t)z * a.P[1] * a.Hpad + kx;
  const int Ny = a.Nout[1];
  C v[A];
#pragma unroll
  for (int r = 0; r < A; ++r) v[r] = valid ? col[(size_t)(t + B * r) * pitch] : mk(T(0), T(0));
  dft_natural<A>(v);
  // the barrier of the hand-off also orders every read of the block's columns
  // before the first row written over them
  col_finish<T, N>(sm, v, b, t, static_cast<const C*>(a.tw_y), [&](int y, C w) {
    if (valid && y < Ny) col[(size_t)y * pitch] = w;
  });
}

template <typename T, int N>
__global__ void __launch_bounds__(ColCfg<T, N>::THREADS, ColCfg<T, N>::MINB) k_gen_z_two(const GenArgs a) {
  gen_z_two_body<T, N>(a, blockIdx.x, blockIdx.y);
}
template <typename T, int N>
__global__ void __launch_bounds__(ColCfg<T, N>::THREADS, ColCfg<T, N>::MINB) k_gen_z_two_batch(const BatchMap m) {
  int loc;
  const GenArgs a = m.args[batch_item(m, &loc)];
  const int gx = (a.Hx + ColCfg<T, N>::LB - 1) / ColCfg<T, N>::LB;
  gen_z_two_body<T, N>(a, loc % gx, loc / gx);
}
template <typename T, int N>
__global__ void __launch_bounds__(ColCfg<T, N>::THREADS, ColCfg<T, N>::MINB) k_mid_y_two(const GenArgs a) {
  mid_y_two_body<T, N>(a, blockIdx.x, blockIdx.y);
}
template <typename T, int N>
__global__ void __launch_bounds__(ColCfg<T, N>::THREADS, ColCfg<T, N>::MINB) k_mid_y_two_batch(const BatchMap m) {
  int loc;
  const GenArgs a = m.args[batch_item(m, &loc)];
  const int gx = (a.Hx + ColCfg<T, N>::LB - 1) / ColCfg<T, N>::LB;
  mid_y_two_body<T, N>(a, loc % gx, loc / gx);
}

}  // namespace scarl
