// c2r_two.cuh -- pass 3 of the padded generator (Hermitian C2R along x, crop,
// blend epilogue) with each line's transform in two in-register stages
// (fft_two.cuh), FP32 and FP64.
//
// L lanes of a warp serve a line, G = 32 / L lines a warp; everything between
// the line's arrival and its last store is warp-local (no block barrier).  The
// raw lines come by bulk asynchronous copies (one per line, per-warp mbarrier,
// bounded wait), stage 1 forms z[k] = (X[k] + X*[N-k]) + i e^{2 pi i k / 2N}
// (X[k] - X*[N-k]) on the way in, stage 2 writes its outputs over the raw line,
// and the epilogue runs with the warp's lanes on consecutive x.  A warp walks
// `two_chunk` groups of lines, so that the block's tables (both twiddle sets,
// s_x and flags) are loaded once for all of them.
#pragma once

#include "c2r_shfl.cuh"
#include "fft_two.cuh"

namespace scarl {

// Factors and lanes of a line of N complex values: stage 1 is B work items of
// DFT-A, stage 2 A items of DFT-B, each taking ceil(items / L) rounds of the
// line's L lanes; the pairs below leave the fewest lanes idle with at most MAXR
// values a lane.
template <typename T, int N> struct TwoLen {
  static constexpr int A = N == 16 ? 4 : N == 24 ? 3 : N == 32 ? 4 : N == 40 ? 5 : N == 48 ? 6 : N == 56 ? 7
                         : N == 64 ? 8 : N == 80 ? 10 : N == 96 ? 12 : N == 112 ? 14 : N == 128 ? 8
                         : N == 160 ? 10 : N == 192 ? 12 : N == 224 ? 14 : N == 256 ? 16 : N == 320 ? 20
                         : N == 384 ? 24 : N == 448 ? 28 : N == 512 ? 16 : N == 640 ? 20 : N == 768 ? 24
                         : N == 896 ? 28 : N == 1024 ? 32 : 1;
  static constexpr int B = N / A;
  static constexpr int L = N >= 512 ? 32 : N >= 128 ? 16 : 8;
  static constexpr int MAXR = sizeof(T) == 4 ? 32 : 16;
  static constexpr bool valid() { return A > 1 && A * B == N && A <= MAXR && B <= MAXR; }
};

template <typename T, int N> struct TwoCfg {
  using Len = TwoLen<T, N>;
  static constexpr int A = Len::A, B = Len::B, L = Len::L, G = 32 / L, WPB = 4, THREADS = 32 * WPB;
  static constexpr int CB = 2 * (int)sizeof(T);  // bytes of a complex value
  static constexpr int LINE_BYTES = ((N + 1) * CB + 15) / 16 * 16;
  static constexpr int XROW = B % 2 == 0 ? B + 1 : B;  // odd: stage 2's reads, rows apart, on distinct banks
  // one round a stage: the hand-off area lies over the raw line, and the outputs
  // over both (every lane reads before any writes); half the shared memory
  static constexpr bool ALIAS = A <= L && B <= L;
  // a line's raw values and its hand-off area; 64 bytes past a multiple of 128
  // where a half-warp holds two lines
  static constexpr int OFF_X = ALIAS ? 0 : (LINE_BYTES + 15) / 16 * 16;
  static constexpr int XB = A * XROW * CB;
  static constexpr int SLOT0 = ALIAS ? ((LINE_BYTES > XB ? LINE_BYTES : XB) + 15) / 16 * 16 : (OFF_X + XB + 15) / 16 * 16;
  static constexpr int SLOT = L == 8 ? SLOT0 + ((64 - SLOT0 % 128) + 128) % 128 : SLOT0;
  static constexpr int OFF_TW = WPB * G * SLOT;          // e^{2 pi i k / 2N}, k < N
  static constexpr int OFF_T2 = OFF_TW + N * CB;         // e^{2 pi i m t / N} at m B + t
  static constexpr int OFF_SX = OFF_T2 + N * CB;         // s_x, x < 2N
  static constexpr int OFF_BAR = OFF_SX + 2 * N * (int)sizeof(T);
  static constexpr int OFF_RED = OFF_BAR + WPB * 8;
  static constexpr int SMEM = OFF_RED + WPB * 16;
  static constexpr int R = A > B ? A : B;
  // registers follow the longer in-register DFT
  static constexpr int MINB = sizeof(T) == 4 ? (R <= 16 ? 7 : R <= 20 ? 6 : R <= 24 ? 5 : 4) : (R <= 12 ? 5 : 4);
  static constexpr bool valid() { return Len::valid() && SMEM <= 200 * 1024; }
};

// Groups of lines a warp walks: up to 8 while about `waves` blocks an SM remain
// (two waves and more, so that the last one is not mostly empty; the large
// tables of long lines want more lines a block).
__host__ __device__ inline int two_chunk(int64_t nlines, int per_block, int N) {
  const int waves = N >= 768 ? 6 : 16;
  const int64_t c = nlines / ((int64_t)per_block * 148 * waves);
  return c < 1 ? 1 : c > 8 ? 8 : (int)c;
}

// e^x in the working precision; FP32: the hardware exponential.
__device__ __forceinline__ float two_exp(float x) { return __expf(x); }
__device__ __forceinline__ double two_exp(double x) { return exp(x); }

// What the blend does along a line, as bounds on x (the flags along an axis are
// an overlap, the inside, an overlap): x < add joins an earlier tile's partial
// sum, x < fin is final (marginal), x < end is this tile's to store.  Three
// compares a point; testing the flag bytes took 24 integer operations an output
// where the crop takes 11.
struct LineBounds {
  int add, fin, end;
};

// K chunks of 32 x values of one line (C2R outputs at ob, destination o, the
// lane's first value x): every read of an earlier tile's partial sum before any
// write.
template <typename T, int K, bool MOM, class Marg>
__device__ __forceinline__ void two_blend(const T* ob, const T* sxs, T* o, int x, const LineBounds& lb, T syz, Marg marg,
                                          double* s1, double* s2) {
  T old[K];
#pragma unroll
  for (int u = 0; u < K; ++u) old[u] = x + 32 * u < lb.add ? o[32 * u] : T(0);
#pragma unroll
  for (int u = 0; u < K; ++u) {
    if (x + 32 * u >= lb.end) continue;
    T w = old[u] + ob[32 * u] * (syz * sxs[32 * u]);
    if (x + 32 * u < lb.fin) {
      w = marg(w);
      if constexpr (MOM) {
        *s1 += (double)w;
        *s2 = fma((double)w, (double)w, *s2);
      }
    }
    o[32 * u] = w;
  }
}
template <typename T, bool MOM>
__device__ __forceinline__ void two_epilogue(const Epilogue& e, const T* ob, const T* sxs, T* o, const LineBounds& lb,
                                             T syz, int lane, double* s1, double* s2) {
  const int marginal = e.marginal;
  const T ms = marginal ? (T)e.ms : T(1), mu = marginal ? (T)e.mmu : T(0);
  auto marg = [&](T v) -> T {
    v = v * ms + mu;
    return marginal == 2 ? two_exp(v) : v;
  };
  if (e.mode == 0) {
#pragma unroll 4
    for (int x = lane; x < lb.end; x += 32) {
      const T w = marg(ob[x]);
      o[x] = w;
      if constexpr (MOM) {
        *s1 += (double)w;
        *s2 = fma((double)w, (double)w, *s2);
      }
    }
    return;
  }
  // groups of four chunks, the rest as one group of four or two
  int x = lane;
#pragma unroll 1
  for (; x - lane + 64 < lb.end; x += 128) two_blend<T, 4, MOM>(ob + x, sxs + x, o + x, x, lb, syz, marg, s1, s2);
  if (x - lane < lb.end) two_blend<T, 2, MOM>(ob + x, sxs + x, o + x, x, lb, syz, marg, s1, s2);
}

template <typename T, int N>
__device__ __forceinline__ void c2r_two_body(const GenArgs& a, int64_t bx) {
  using Cfg = TwoCfg<T, N>;
  using C = cplx_t<T>;
  constexpr int A = Cfg::A, B = Cfg::B, L = Cfg::L, G = Cfg::G;
  extern __shared__ __align__(128) unsigned char two_sm[];
  const int warp = (int)threadIdx.x >> 5, lane = (int)threadIdx.x & 31;
  const int li = lane / L, t0 = lane % L;
  unsigned char* wreg = two_sm + warp * G * Cfg::SLOT;
  C* tws = reinterpret_cast<C*>(two_sm + Cfg::OFF_TW);
  C* tw2 = reinterpret_cast<C*>(two_sm + Cfg::OFF_T2);
  T* sxs = reinterpret_cast<T*>(two_sm + Cfg::OFF_SX);
  const uint32_t bar = tc::smem_u32(two_sm + Cfg::OFF_BAR + warp * 8);
  const int Nx = a.Nout[0], Ny = a.Nout[1];
  const int nlines = Ny * a.Nout[2];  // at most 2048^2
  const int chunk = two_chunk(nlines, Cfg::WPB * G, N);
  const int l00 = ((int)bx * chunk * Cfg::WPB + warp) * G;  // the warp's first line; its groups are WPB G apart
  const bool blend = a.epi.mode != 0;
  // the group's lines: bulk copies issued by lane 0, or, for a caller without a
  // status word to report an expired wait in, 16-byte cp.async by every lane
  const bool bulk = a.status != nullptr;
  auto fetch = [&](int l0) {
    const int nv = min(G, nlines - l0);
    const C* work = static_cast<const C*>(a.work);
    if (bulk && lane == 0) mbar_expect_tx(bar, (uint32_t)(nv * Cfg::LINE_BYTES));
    for (int i = 0; i < nv; ++i) {
      const int l = l0 + i, z = l / Ny, y = l - z * Ny;
      const C* src = work + ((size_t)z * a.P[1] + (size_t)y) * a.Hpad;
      unsigned char* dst = wreg + i * Cfg::SLOT;
      if (!bulk) {
        for (int c = lane; c < Cfg::LINE_BYTES / 16; c += 32)
          cp_async16(dst + 16 * c, reinterpret_cast<const char*>(src) + 16 * c);
      } else if (lane == 0) {
        bulk_g2s(tc::smem_u32(dst), src, Cfg::LINE_BYTES, bar);
      }
    }
  };
  if (lane == 0) tc::mbar_init(bar, 1);
  if (l00 < nlines) fetch(l00);
  {
    const C* twx = static_cast<const C*>(a.tw_x);
    for (int i = (int)threadIdx.x; i < N; i += Cfg::THREADS) {
      tws[i] = __ldg(twx + i);
      tw2[i] = __ldg(twx + 2 * (i / B) * (i % B));
    }
    if (blend) {
      const T* sx = sw_of<T>(a.epi.ax[0]);
      for (int i = (int)threadIdx.x; i < Nx; i += Cfg::THREADS) sxs[i] = a.epi.apply_pou ? __ldg(sx + i) : T(1);
    }
  }
  __syncthreads();  // tables and the warps' barrier initialisation
  double s1 = 0.0, s2 = 0.0;
  const bool mom = a.epi.mom != nullptr;
  uint32_t phase = 0;
#pragma unroll 1
  for (int c = 0; c < chunk; ++c) {
    const int l0 = l00 + c * Cfg::WPB * G;
    if (l0 >= nlines) break;
    if (!bulk) {
      cp_async_wait_all();
      __syncwarp();
    } else if (!warp_bulk_wait(bar, phase, lane, a.wait_test)) {
      // a copy did not land in time: report, give it one more bounded wait
      // (the copies write this block's shared memory), leave the rest
      if (lane == 0) {
        atomicOr(a.status, 1);
        tc::mbar_wait(bar, phase, kBulkWaitNs);
      }
      __syncwarp();
      break;
    }
    phase ^= 1;
    C* line = reinterpret_cast<C*>(wreg + li * Cfg::SLOT);
    C* xch = reinterpret_cast<C*>(wreg + li * Cfg::SLOT + Cfg::OFF_X);
    auto load1 = [&](int t, C* v) {  // pre-combination and DFT-A of work item t
#pragma unroll
      for (int r = 0; r < A; ++r) {
        const int k = t + B * r;
        const C xk = line[k], xn = line[N - k];
        const C xc = cconj(xn);
        const C e = cadd(xk, xc);
        const C o = cmul(csub(xk, xc), tws[k]);
        C z = mk(e.x - o.y, e.y + o.x);
        if (r == 0 && t == 0) z = mk(xk.x + xn.x, xk.x - xn.x);
        v[r] = z;
      }
      dft_natural<A>(v);
#pragma unroll
      for (int m = 1; m < A; ++m) v[m] = cmul(v[m], tw2[m * B + t]);
    };
    auto store1 = [&](int t, const C* v) {
#pragma unroll
      for (int m = 0; m < A; ++m) xch[m * Cfg::XROW + t] = v[m];
    };
    auto load2 = [&](int m, C* v) {
#pragma unroll
      for (int t = 0; t < B; ++t) v[t] = xch[m * Cfg::XROW + t];
      dft_natural<B>(v);
    };
    auto store2 = [&](int m, const C* v) {  // outputs y[m + A s]: reals 2n, 2n + 1
#pragma unroll
      for (int s = 0; s < B; ++s) line[m + A * s] = v[s];
    };
    if constexpr (Cfg::ALIAS) {
      {
        C v[A];
        if (t0 < B) load1(t0, v);
        __syncwarp();
        if (t0 < B) store1(t0, v);
      }
      __syncwarp();
      {
        C v[B];
        if (t0 < A) load2(t0, v);
        __syncwarp();
        if (t0 < A) store2(t0, v);
      }
    } else {
#pragma unroll 1
      for (int t = t0; t < B; t += L) {
        C v[A];
        load1(t, v);
        store1(t, v);
      }
      __syncwarp();
#pragma unroll 1
      for (int m = t0; m < A; m += L) {
        C v[B];
        load2(m, v);
        store2(m, v);
      }
    }
    __syncwarp();
    // ---- epilogue: one line at a time, lanes along x; lane i < G holds what
    //      line i needs ----
    long long base = 0;
    int yz = 0;  // bit 0: contributes, bit 1: not the first, bit 2: the last
    T syz = T(1);
    if (lane < G && l0 + lane < nlines) {
      const int l = l0 + lane, z = l / Ny, y = l - z * Ny;
      const Epilogue& e = a.epi;
      if (!blend) {
        base = (long long)Nx * l;
        yz = 5;
      } else {
        base = e.off[0] + e.L[0] * ((e.off[1] + y) + e.L[1] * (e.off[2] + z));
        yz = (y < e.ax[1].end && z < e.ax[2].end ? 1 : 0) | (y < e.ax[1].add || z < e.ax[2].add ? 2 : 0) |
             (y < e.ax[1].fin && z < e.ax[2].fin ? 4 : 0);
        if (e.apply_pou) syz = sw_of<T>(e.ax[1])[y] * sw_of<T>(e.ax[2])[z];
      }
    }
    const LineBounds xb = blend ? LineBounds{a.epi.ax[0].add, a.epi.ax[0].fin, a.epi.ax[0].end} : LineBounds{0, Nx, Nx};
#pragma unroll 1
    for (int i = 0; i < G; ++i) {
      if (l0 + i >= nlines) break;
      T* o = static_cast<T*>(a.epi.out) + __shfl_sync(0xffffffffu, base, i);
      const int fi = __shfl_sync(0xffffffffu, yz, i);
      const T si = __shfl_sync(0xffffffffu, syz, i);
      if (!(fi & 1)) continue;
      const LineBounds lb{(fi & 2) ? xb.end : min(xb.add, xb.end), (fi & 4) ? min(xb.fin, xb.end) : 0, xb.end};
      const T* ob = reinterpret_cast<const T*>(wreg + i * Cfg::SLOT);
      if (mom) two_epilogue<T, true>(a.epi, ob, sxs, o, lb, si, lane, &s1, &s2);
      else two_epilogue<T, false>(a.epi, ob, sxs, o, lb, si, lane, &s1, &s2);
    }
    __syncwarp();
    if (c + 1 < chunk && l0 + Cfg::WPB * G < nlines) {
      if (lane == 0) tc::fence_smem_to_async();  // the warp's reads and writes before the copies'
      fetch(l0 + Cfg::WPB * G);
    }
  }
  if (mom) {  // the block's pair: warps in shared memory, then thread 0
    double* red = reinterpret_cast<double*>(two_sm + Cfg::OFF_RED);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      s1 += __shfl_xor_sync(0xffffffffu, s1, o);
      s2 += __shfl_xor_sync(0xffffffffu, s2, o);
    }
    if (lane == 0) {
      red[2 * warp] = s1;
      red[2 * warp + 1] = s2;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      double u1 = 0.0, u2 = 0.0;
#pragma unroll
      for (int w = 0; w < Cfg::WPB; ++w) {
        u1 += red[2 * w];
        u2 += red[2 * w + 1];
      }
      a.epi.mom[2 * bx] = u1;
      a.epi.mom[2 * bx + 1] = u2;
    }
  }
}

template <typename T, int N>
__global__ void __launch_bounds__(TwoCfg<T, N>::THREADS, TwoCfg<T, N>::MINB) k_c2r_x_two(const GenArgs a) {
  c2r_two_body<T, N>(a, blockIdx.x);
}
template <typename T, int N>
__global__ void __launch_bounds__(TwoCfg<T, N>::THREADS, TwoCfg<T, N>::MINB) k_c2r_x_two_batch(const BatchMap m) {
  int loc;
  const GenArgs a = m.args[batch_item(m, &loc)];
  c2r_two_body<T, N>(a, loc);
}

}  // namespace scarl
