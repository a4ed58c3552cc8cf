// stats.cu -- directional covariance estimator of Stat_ScaRL
// (SRC_F/Stat_ScaRL/statistics_RF.f90:258-462, rebuild_Sk_FFT) in FP64.  The
// reference forms |FFT(t)/n|^2 per line, averages over the other two axes and
// inverts: that is the circular autocorrelation
//   Sk[m] = 1/(n * nlines) * sum_lines sum_i t_i t_{(i+m) mod n},
//   t = ((x - avg) / std) * w (Tukey window along the line),
// here from the linear lag sums R(j) = sum_i t_i t_{i+j}, Sk[m] ~ R(m) + R(n-m),
// so that any line length runs on power-of-two transforms: with lines
// zero-padded to N >= 2n - 2, sum_k |Z_k|^2 e^{-2 pi i k j / N} / N = R(j) +
// R(N - j), and the second term is zero for j < n except R(n - 1) again at
// N = 2n - 2.
//
// Two real lines share one complex transform, z = a + i b: the real part of
// z's autocorrelation is the sum of theirs, so the powers |Z_k|^2 are summed
// as they leave the last stage, each thread keeping its own bins in FP64
// registers over all its lines: no even/odd split, nothing written per line.
#include <algorithm>

#include "fft_engine.cuh"
#include "scarl_internal.h"

namespace scarl {

namespace {

// 16 values a thread (radix 16 stages); 256 threads a block, at most 32 pairs
// of lines (fewer lanes than that on one row do not fill the loads' sectors)
constexpr int kPowE = 16;
template <typename T, int N> struct PowCfg {
  static constexpr int TPL = N / kPowE;
  static constexpr int B = TPL >= 256 ? 1 : (256 / TPL > 32 ? 32 : 256 / TPL);
  static constexpr int NT = B * TPL;
  static constexpr int LS = line_slots<N, kPowE>();
  static constexpr int PRE = 18 * NT * (int)sizeof(T);  // the next lines' values, 2 x 9 a thread
  // twiddles in shared memory where two blocks an SM keep their place
  static constexpr bool TWS = B * LS * 16 + PRE + N * 16 <= 113 * 1024;
  static constexpr int SMEM = (B * LS + (TWS ? N : 0)) * 16 + PRE;
  static constexpr int MINB = NT >= 512 ? 1 : 512 / NT;  // 128 registers a thread
};

struct PowGeom {
  const void* f;
  int n;            // points a line
  int na;           // lines along the fastest other axis
  int64_t sa, sb;   // element strides of the other axes
  int64_t st;       // element stride along the line
  int64_t nlines;
  double avg;
  const double* win;  // n
  const double2* tw;  // e^{2 pi i m / N}, m < N
  double* partial;    // gridDim.x * N
};

// What bounds it: the shared-memory pipe (two hand-offs of 16-byte values a
// transform), then FP64.  The next group's values come by cp.async into each
// thread's own slots while the current group is transformed; loaded
// when needed they left the block waiting on memory (513 x 512 x 256 FP32
// points: 593 / 482 / 483 us along x / y / z, now 409 / 409 / 323; the direct
// lag sums that this replaces took 36.6 ms on 513^3 points, all axes, this
// 2.6 ms).
template <typename T> __device__ __forceinline__ void cp_own(T* dst, const T* src) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(s), "l"(src), "n"(sizeof(T)) : "memory");
}

template <typename T, int N, bool ROW>
__global__ void __launch_bounds__(PowCfg<T, N>::NT, PowCfg<T, N>::MINB > 16 ? 16 : PowCfg<T, N>::MINB)
    k_line_power(const PowGeom g) {
  using Cfg = PowCfg<T, N>;
  constexpr int TPL = Cfg::TPL, B = Cfg::B, LS = Cfg::LS;
  // lanes along the line only for short x lines: from N = 512 on, lanes across
  // lines give the stages conflict-free twiddle reads and still load whole
  // sectors (n = 400 x 316 x 316 points, three axes: 0.943 against 1.033 ms; at
  // N = 128, FP64: 1.42 against 1.49 ms the other way)
  constexpr bool ALONG = ROW && N < 512;
  constexpr SmemOrder O = ALONG ? SmemOrder::LineFast : SmemOrder::BatchFast;
  extern __shared__ __align__(16) unsigned char pow_sm[];
  double2* sm = reinterpret_cast<double2*>(pow_sm);
  const int b = ALONG ? (int)threadIdx.x / TPL : (int)threadIdx.x % B;
  const int t = ALONG ? (int)threadIdx.x % TPL : (int)threadIdx.x / B;
  const T* f = static_cast<const T*>(g.f);
  const double2* tw = g.tw;
  if constexpr (Cfg::TWS) {
    double2* tws = sm + B * LS;
    for (int i = (int)threadIdx.x; i < N; i += Cfg::NT) tws[i] = __ldg(g.tw + i);
    __syncthreads();
    tw = tws;
  }
  constexpr int RL = last_radix<N, kPowE>();
  double acc[kPowE];
#pragma unroll
  for (int i = 0; i < kPowE; ++i) acc[i] = 0.0;
  const int64_t npairs = (g.nlines + 1) / 2, ngroups = (npairs + B - 1) / B;
  T* pre = reinterpret_cast<T*>(pow_sm + (size_t)(B * LS + (Cfg::TWS ? N : 0)) * 16) + threadIdx.x;
  // inputs i = t + r N / 16 (the thread's one first-stage butterfly); n <=
  // N / 2 + 1, so r > 8 is zero.  Slots 2 r, 2 r + 1 hold lines l, l + 1.
  auto fetch = [&](int64_t grp) {
    const int64_t l = 2 * (grp * B + b);
    const bool v0 = l < g.nlines, v1 = l + 1 < g.nlines;
    const T* p0 = f + (v0 ? (l % g.na) * g.sa + (l / g.na) * g.sb : 0) + t * g.st;
    const T* p1 = f + (v1 ? ((l + 1) % g.na) * g.sa + ((l + 1) / g.na) * g.sb : 0) + t * g.st;
#pragma unroll
    for (int r = 0; r < 9; ++r)
      if (t + r * (N / 16) < g.n) {
        if (v0) cp_own(pre + (2 * r) * Cfg::NT, p0 + r * (N / 16) * g.st);
        if (v1) cp_own(pre + (2 * r + 1) * Cfg::NT, p1 + r * (N / 16) * g.st);
      }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  fetch(blockIdx.x);
  for (int64_t grp = blockIdx.x; grp < ngroups; grp += gridDim.x) {
    const int64_t l = 2 * (grp * B + b);
    const bool v0 = l < g.nlines, v1 = l + 1 < g.nlines;
    auto load = [&](int j, double2* v) {
      asm volatile("cp.async.wait_all;\n" ::: "memory");
#pragma unroll
      for (int r = 0; r < 16; ++r) {
        const int i = j + r * (N / 16);
        if (r > 8 || i >= g.n) {
          v[r] = make_double2(0.0, 0.0);
          continue;
        }
        const double w = __ldg(g.win + i);
        v[r] = make_double2(v0 ? ((double)pre[(2 * r) * Cfg::NT] - g.avg) * w : 0.0,
                            v1 ? ((double)pre[(2 * r + 1) * Cfg::NT] - g.avg) * w : 0.0);
      }
      if (grp + gridDim.x < ngroups) fetch(grp + gridDim.x);
    };
    auto store = [&](int j, const double2* o) {
      const int q = (j - t) / TPL;
#pragma unroll
      for (int r = 0; r < RL; ++r) acc[q * RL + r] = fma(o[r].x, o[r].x, fma(o[r].y, o[r].y, acc[q * RL + r]));
    };
    line_ifft<double2, N, kPowE, O, B, LS>(sm, b, t, tw, load, store);
  }
  __syncthreads();
  // bins summed over the block's lines, in line order
  double* red = reinterpret_cast<double*>(pow_sm);
#pragma unroll
  for (int q = 0; q < kPowE / RL; ++q)
#pragma unroll
    for (int r = 0; r < RL; ++r) red[b * N + t + TPL * q + r * (N / RL)] = acc[q * RL + r];
  __syncthreads();
  for (int k = (int)threadIdx.x; k < N; k += Cfg::NT) {
    double s = 0.0;
#pragma unroll 4
    for (int bb = 0; bb < B; ++bb) s += red[bb * N + k];
    g.partial[(int64_t)blockIdx.x * N + k] = s;
  }
}

template <typename T, int N, bool ROW>
cudaError_t run_line_power(const PowGeom& g, int want, int* blocks, cudaStream_t s) {
  using Cfg = PowCfg<T, N>;
  auto kern = k_line_power<T, N, ROW>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM);
  if (e != cudaSuccess) return e;
  if (blocks) {
    int per_sm = 0, dev = 0, sms = 148;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, Cfg::NT, Cfg::SMEM)) != cudaSuccess) return e;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int64_t ngroups = ((g.nlines + 1) / 2 + Cfg::B - 1) / Cfg::B;
    *blocks = (int)std::max<int64_t>(1, std::min<int64_t>(ngroups, (int64_t)std::max(per_sm, 1) * sms));
    return cudaSuccess;
  }
  kern<<<want, Cfg::NT, Cfg::SMEM, s>>>(g);
  return cudaGetLastError();
}

template <typename T, bool ROW>
cudaError_t line_power_n(int N, const PowGeom& g, int want, int* blocks, cudaStream_t s) {
  switch (N) {
    case 16: return run_line_power<T, 16, ROW>(g, want, blocks, s);
    case 32: return run_line_power<T, 32, ROW>(g, want, blocks, s);
    case 64: return run_line_power<T, 64, ROW>(g, want, blocks, s);
    case 128: return run_line_power<T, 128, ROW>(g, want, blocks, s);
    case 256: return run_line_power<T, 256, ROW>(g, want, blocks, s);
    case 512: return run_line_power<T, 512, ROW>(g, want, blocks, s);
    case 1024: return run_line_power<T, 1024, ROW>(g, want, blocks, s);
    case 2048: return run_line_power<T, 2048, ROW>(g, want, blocks, s);
    case 4096: return run_line_power<T, 4096, ROW>(g, want, blocks, s);
    case 8192: return run_line_power<T, 8192, ROW>(g, want, blocks, s);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t line_power(int dt, const void* f, const int L[3], int dir, int N, double avg, const double* win,
                       const void* tw, double* partial, int want, int* blocks, cudaStream_t s) {
  PowGeom g;
  g.f = f;
  g.n = L[dir];
  g.avg = avg;
  g.win = win;
  g.tw = static_cast<const double2*>(tw);
  g.partial = partial;
  const int64_t L0 = L[0], L1 = L[1], L2 = L[2];
  g.na = dir == 0 ? L[1] : L[0];
  g.sa = dir == 0 ? L0 : 1;
  g.sb = dir == 2 ? L0 : L0 * L1;
  g.st = dir == 0 ? 1 : dir == 1 ? L0 : L0 * L1;
  g.nlines = dir == 0 ? L1 * L2 : dir == 1 ? L0 * L2 : L0 * L1;
  if (g.n > N / 2 + 1) return cudaErrorInvalidValue;
  if (dt == 8)
    return dir == 0 ? line_power_n<double, true>(N, g, want, blocks, s) : line_power_n<double, false>(N, g, want, blocks, s);
  return dir == 0 ? line_power_n<float, true>(N, g, want, blocks, s) : line_power_n<float, false>(N, g, want, blocks, s);
}

// Sum of the rows of partial (nrows x nbins): 32 bins a block, 32 groups of
// rows summed side by side (a bin a thread took 34 us for 296 rows of 769
// bins, a chain of dependent loads; this 5).
__global__ void __launch_bounds__(1024) k_bins(const double* __restrict__ partial, int nrows, int nbins,
                                               double* __restrict__ bins) {
  __shared__ double red[32][33];
  const int c = threadIdx.x & 31, w = threadIdx.x >> 5, k = (int)blockIdx.x * 32 + c;
  double s = 0.0;
  if (k < nbins)
#pragma unroll 4
    for (int r = w; r < nrows; r += 32) s += partial[(int64_t)r * nbins + k];
  red[w][c] = s;
  __syncthreads();
  s = red[c][w];
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if (c == 0 && (int)blockIdx.x * 32 + w < nbins) bins[(int)blockIdx.x * 32 + w] = s;
}

// S(j) = (1/N) sum_k P_k cos(2 pi k j / N), one block a lag.
__global__ void __launch_bounds__(256) k_power_lags(const double* __restrict__ bins, int N, const double2* __restrict__ tw,
                                                    double* __restrict__ S) {
  const int j = blockIdx.x;
  double s = 0.0;
  for (int k = threadIdx.x; k < N; k += 256) s = fma(bins[k], tw[(int)((int64_t)k * j & (N - 1))].x, s);
  __shared__ double red[8];
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    s = 0.0;
    for (int i = 0; i < 8; ++i) s += red[i];
    S[j] = s / (double)N;
  }
}

}  // namespace

int line_power_length(int n) {
  int N = 16;
  while (N < 2 * n - 2) N <<= 1;
  return N <= 8192 ? N : 0;
}

int line_power_blocks(int dt, const int L[3], int dir, int N) {
  int nb = -1;
  if (line_power(dt, nullptr, L, dir, N, 0.0, nullptr, nullptr, nullptr, 0, &nb, nullptr) != cudaSuccess) {
    cudaGetLastError();
    return -1;
  }
  return nb;
}

cudaError_t launch_line_power(int dt, const void* f, const int L[3], int dir, int N, double avg, const double* win,
                              const void* tw, double* partial, int nblocks, double* bins, double* S, cudaStream_t s) {
  cudaError_t e = line_power(dt, f, L, dir, N, avg, win, tw, partial, nblocks, nullptr, s);
  if (e != cudaSuccess) return e;
  if ((e = launch_bins(partial, nblocks, N, bins, s)) != cudaSuccess) return e;
  k_power_lags<<<L[dir], 256, 0, s>>>(bins, N, static_cast<const double2*>(tw), S);
  return cudaGetLastError();
}

cudaError_t launch_bins(const double* partial, int nrows, int nbins, double* bins, cudaStream_t s) {
  k_bins<<<(nbins + 31) / 32, 1024, 0, s>>>(partial, nrows, nbins, bins);
  return cudaGetLastError();
}

// Sum of n FP64 pairs (x, y) into out[0], out[1] in a fixed order: block b
// sums the pairs b, b + gridDim.x, ... (each thread a fixed stride, then a
// fixed tree) into part[b]; one block then sums the gridDim.x parts.
constexpr int kPairBlocks = 148;
__device__ __forceinline__ void pair_tree(double a, double b, double* out) {
  __shared__ double r0[256], r1[256];
  r0[threadIdx.x] = a;
  r1[threadIdx.x] = b;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) {
      r0[threadIdx.x] += r0[threadIdx.x + w];
      r1[threadIdx.x] += r1[threadIdx.x + w];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    out[0] = r0[0];
    out[1] = r1[0];
  }
}
__global__ void __launch_bounds__(256) k_pair_part(const double* __restrict__ p, int64_t n,
                                                   double* __restrict__ part) {
  double a = 0.0, b = 0.0;
  for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < n; i += (int64_t)gridDim.x * 256) {
    a += p[2 * i];
    b += p[2 * i + 1];
  }
  pair_tree(a, b, part + 2 * blockIdx.x);
}
__global__ void __launch_bounds__(256) k_pair_final(const double* __restrict__ part, int nparts,
                                                    double* __restrict__ out) {
  double a = 0.0, b = 0.0;
  for (int i = threadIdx.x; i < nparts; i += 256) {
    a += part[2 * i];
    b += part[2 * i + 1];
  }
  pair_tree(a, b, out);
}

// part: 2 kPairBlocks doubles of scratch.
cudaError_t launch_pair_sum(const double* pairs, int64_t n, double* part, double* out, cudaStream_t s) {
  k_pair_part<<<kPairBlocks, 256, 0, s>>>(pairs, n, part);
  k_pair_final<<<1, 256, 0, s>>>(part, kPairBlocks, out);
  return cudaGetLastError();
}
int pair_sum_parts() { return kPairBlocks; }

}  // namespace scarl
