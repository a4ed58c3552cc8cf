// dct_literal.cu -- the reference's active generator, gen_std_gauss_FFT
// (SRC_F/fftw_ScaRL.f90:261-418), in FP64, for a batch of tiles of one shape:
//   k_dct_spec : Sk = gamma * sqrt(prod_d corrL_d exp(-PI k_d^2)) * cos(2 PI phi)
//                on the (Np/2)^3 octant (the rest of the reference's array is
//                uninitialised; it is zero here and never stored).
//   k_dct_mm   : unnormalised DCT-III (FFTW REDFT01) along one axis,
//                y_n = sum_i c_i x_i cos(pi i (2n+1) / (2N)), c_0 = 1, c_i = 2,
//                over the octant's nonzero inputs, as a matrix product on the
//                FP64 tensor cores.  Three launches (x, y, z) form the 3D
//                transform of fftw_plan_r2r_3d(REDFT01 x3).
//
// Folding: cos(pi i (2(N-1-n)+1) / (2N)) = (-1)^i cos(pi i (2n+1) / (2N)), so
// with E and O the sums over even and odd i, y_n = E_n + O_n and
// y_{N-1-n} = E_n - O_n: half the products of the plain sum.
//
// Every axis is one form, D[m][n] = sum_k A[k][m] B[k][n] with both operands
// stored row by row of k (16-byte copies, no transposition):
//   x: A = spectrum [i][line], B = cosines [i][n]; D = rows of x
//   y: A = cosines [j][n], B = rows of x per kz
//   z: A = cosines [k][n], B = whole planes; D goes through the output stage
//      (crop, or partition of unity, overlap sum and marginal into the field)
// The spectrum is written line-fastest for that, and rows are padded to even
// lengths so that every copy starts on 16 bytes.
//
// What bounds it: the FP64 tensor pipe, 42-60 % busy (45 % in the z step of a
// 297 x 277 x 267 tile, whose output stage takes the rest).  mma.sync f64
// (DMMA) runs at 37.0 TFLOP/s on B200 where independent FMAs reached 27.9 in
// the same loop, and takes its operands from a quarter of the shared-memory
// reads.  A 64 x 64 tile of both parities per 256-thread block (32 accumulators
// a thread, two blocks an SM); 32-row tiles with three blocks an SM measured
// the same (3.20 against 3.17 ms).  Measured on the 513^3 deck (8 such tiles,
// blend included): 3.17 ms, 9.87 ms with plain 4 x 4 register tiles, unfolded
// sums and a separate blend pass.
#include <algorithm>
#include <type_traits>

#include "epilogue.cuh"
#include "scarl_common.cuh"
#include "scarl_internal.h"

namespace scarl {

constexpr double kPiRefD = 3.1415926535898;  // SRC_F/constants_ScaRL.f90:5

// One thread per mode: blockIdx.x * 128 + threadIdx.x is the line l = j + K1 k,
// blockIdx.z the tile, i walks from blockIdx.y by gridDim.y (at most 65535; an
// axis may have more inputs).
__global__ void __launch_bounds__(128) k_dct_spec(const DctArgs a) {
  const int nl = a.K[1] * a.K[2], l = (int)(blockIdx.x * 128 + threadIdx.x);
  if (l >= nl) return;
  const int tile = blockIdx.z, k = l / a.K[1], j = l - k * a.K[1];
  for (int i = blockIdx.y; i < a.K[0]; i += gridDim.y) {
    const double* cx = a.cexp + (int64_t)tile * (a.K[0] + a.K[1] + a.K[2]);
    const double* cy = cx + a.K[0];
    const double* cz = cy + a.K[1];
    const int64_t o = i + (int64_t)a.K[0] * l, n = (int64_t)a.K[0] * nl;  // the reference's element order
    double S = 1.0;
    S = __dmul_rn(__dmul_rn(S, a.corrL[0]), cx[i]);
    S = __dmul_rn(__dmul_rn(S, a.corrL[1]), cy[j]);
    S = __dmul_rn(__dmul_rn(S, a.corrL[2]), cz[k]);
    double phi;
    if (a.phi) {
      phi = a.phi[tile * n + o];
    } else {
      const u32x4 q = philox4x32_10({(uint32_t)o, (uint32_t)((uint64_t)o >> 32), a.stream, 1u},
                                    a.k0 + (uint32_t)tile, a.k1);
      phi = u01_d(q.x, q.y);
    }
    const double g = a.gamma ? a.gamma[tile * n + o] : 1.0;
    const double c = cos(__dmul_rn(__dmul_rn(2.0, kPiRefD), phi));
    a.sk[((int64_t)tile * a.K[0] + i) * a.lp + l] = __dmul_rn(__dmul_rn(g, sqrt(S)), c);
  }
}

// tab[i][n] = c_i cos(pi i (2n + 1) / (2N)), i < K, n < H = (N + 1) / 2, rows
// hp apart, the angle index reduced exactly (ctab[m] = cos(pi m / (2N)), m < 4N).
__global__ void k_dct_table(const double* __restrict__ ctab, int N, int K, int H, int hp, double* __restrict__ tab) {
  const int64_t n = (int64_t)K * hp;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = t / hp, c = t - i * hp;
    const int64_t m = (i * (2 * c + 1)) % (4 * (int64_t)N);
    tab[t] = c < H ? (i == 0 ? 1.0 : 2.0 * ctab[m]) : 0.0;
  }
}

// The same value formed in the kernel, for axes whose matrix would be too large
// to keep: x mod 4 N by Barrett's reduction, inv = floor((2^64 - 1) / 4 N) (the
// quotient comes out right or one short).
__device__ __forceinline__ double dct_cosine(const double* __restrict__ ctab, int N, uint64_t inv, int i, int c) {
  if (c >= (N + 1) / 2) return 0.0;
  if (i == 0) return 1.0;
  const uint64_t d = 4 * (uint64_t)N, x = (uint64_t)i * (uint64_t)(2 * (int64_t)c + 1);
  uint64_t m = x - __umul64hi(x, inv) * d;
  if (m >= d) m -= d;
  return 2.0 * __ldg(ctab + m);
}

cudaError_t launch_dct_table(const double* ctab, int N, int K, double* tab, cudaStream_t s) {
  const int H = (N + 1) / 2, hp = (H + 1) / 2 * 2;
  const int64_t n = (int64_t)K * hp;
  k_dct_table<<<(unsigned)std::min<int64_t>((n + 255) / 256, 148 * 16), 256, 0, s>>>(ctab, N, K, H, hp, tab);
  return cudaGetLastError();
}

// One axis: batch element b takes A + b bA, B + b bB, D + b bD.
struct DctMM {
  const double* A;
  const double* B;
  double* D;
  const double* ctab;     // cos(pi m / (2 Nfull)) where the cosine operand is formed from it, else null
  uint64_t inv;           // of 4 Nfull (dct_cosine)
  int64_t lda, ldb, ldd;  // row strides (elements, even for A and B)
  int64_t bA, bB, bD;
  int wa, wb;             // readable elements of a row of A and B (even)
  int M, N, K, Nfull;     // rows and columns of D (before folding), inputs, transform length
  int nm, nn, batch;      // row and column tiles, batch elements
  int n0, n0p, n1;        // final stage: column c = x + n0p y, x < n0, y < n1
  Epilogue epi;           // final stage
};

constexpr int kMmNT = 64, kMmKB = 8, kMmStages = 3;
template <int MW> struct MmCfg {
  static constexpr int MT = 16 * MW;
  // row strides of 4 mod 16 elements: the 4 x 8 fragment reads of a warp fall
  // on distinct banks
  static constexpr int SA = MT + 4, SB = kMmNT + 4;
  static constexpr int STAGE = 2 * kMmKB * (SA + SB);  // doubles: both parities
  static constexpr int SO = kMmNT + 8;  // output staging row: 16-byte stores of 8 x 4 lanes on distinct banks
  static constexpr int OFF_OUT = kMmStages * STAGE;
  static constexpr int SMEM = (OFF_OUT + MT * SO) * 8;
};

__device__ __forceinline__ void cp16_zfill(unsigned dst, const double* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void dmma(double (&c0)[2], double (&c1)[2], const double (&a)[4], double b0, double b1) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
               : "+d"(c0[0]), "+d"(c0[1]), "+d"(c1[0]), "+d"(c1[1])
               : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b0), "d"(b1));
}

// MM_FINAL_EXP: the output stage with a lognormal marginal (exp in code of its
// own: inlined beside the affine one it is evaluated for both)
enum MmOut { MM_FOLD_N, MM_FOLD_M, MM_FINAL, MM_FINAL_EXP };

// Tiles of MT x 64 of both parities' products, blocks walking them with the
// next tile's first copies in flight during the current tile's output.  Warps:
// 2 along m (interleaved groups of 16 rows, so that a partial last tile keeps
// both busy) x 4 along n.
// ROOTS: the cosine operand (B in the x step, A in the others) is formed from
// p.ctab instead of copied.
template <int MW, int OUT, bool ROOTS>
__global__ void __launch_bounds__(256, 2) k_dct_mm(const DctMM p) {
  using Cfg = MmCfg<MW>;
  constexpr bool COS_A = ROOTS && OUT != MM_FOLD_N, COS_B = ROOTS && OUT == MM_FOLD_N;
  constexpr bool EXP = OUT == MM_FINAL_EXP;
  extern __shared__ __align__(16) double mm_sm[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int wm = warp >> 2, wn = warp & 3, g = lane >> 2, t = lane & 3;
  const unsigned total = (unsigned)p.nm * p.nn * p.batch;
  const int nk = (p.K + 2 * kMmKB - 1) / (2 * kMmKB);

  // A stage holds 16 inputs i (rows in input order: parity alternates), each a
  // row of MT / 2 chunks of A and 32 of B; this thread copies chunk qa of rows
  // ra + RA u and chunk qb of rows rb + 8 u (RA is even: a thread's rows share
  // their parity).  Inputs beyond K and columns beyond the row are zero.
  constexpr int CA = Cfg::MT / 2, RA = 256 / CA, UA = 2 * kMmKB / RA;
  static_assert(RA % 2 == 0 && UA >= 1, "copies per thread");
  const int qa = 2 * (tid % CA), ra = tid / CA, qb = 2 * (tid % 32), rb = tid / 32;
  const unsigned sm0 = (unsigned)__cvta_generic_to_shared(mm_sm);
  auto slot_row = [](int row, int ld) { return ((row & 1) * kMmKB + (row >> 1)) * ld; };
  const unsigned da = sm0 + 8 * (slot_row(ra, Cfg::SA) + qa);
  const unsigned db = sm0 + 8 * (2 * kMmKB * Cfg::SA + slot_row(rb, Cfg::SB) + qb);
  const double *pa = nullptr, *pb = nullptr;
  int ka = 0, kb_ = 0;
  int m0n = 0, n0n = 0;
  unsigned btn = 0;
  auto load = [&](int kb, int slot) {
    const int i0 = 2 * kMmKB * kb;
    const unsigned so = slot * (Cfg::STAGE * 8);
#pragma unroll
    for (int u = 0; u < UA; ++u) {
      if constexpr (COS_A) continue;
      const bool ok = i0 + RA * u < ka;
      cp16_zfill(da + so + 8 * (RA / 2) * Cfg::SA * u, ok ? pa + (int64_t)(RA * u) * p.lda : p.A, ok ? 16 : 0);
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      if constexpr (COS_B) continue;
      const bool ok = i0 + 8 * u < kb_;
      cp16_zfill(db + so + 8 * 4 * Cfg::SB * u, ok ? pb + (int64_t)(8 * u) * p.ldb : p.B, ok ? 16 : 0);
    }
    pa += 2 * kMmKB * p.lda;
    pb += 2 * kMmKB * p.ldb;
  };
  // ROOTS: the thread's cosines of a stage, in registers until the current stage
  // has been multiplied
  constexpr int UC = !ROOTS ? 1 : COS_A ? UA : 2;
  double2 cosv[UC];
  auto form = [&](int kb) {
#pragma unroll
    for (int u = 0; u < (ROOTS ? UC : 0); ++u) {
      const int i = 2 * kMmKB * kb + (COS_A ? ra + RA * u : rb + 8 * u), c = COS_A ? m0n + qa : n0n + qb;
      cosv[u] = i < p.K ? make_double2(dct_cosine(p.ctab, p.Nfull, p.inv, i, c), dct_cosine(p.ctab, p.Nfull, p.inv, i, c + 1))
                        : make_double2(0.0, 0.0);
    }
  };
  auto put = [&](int slot) {
    double* st = mm_sm + slot * Cfg::STAGE + (COS_A ? slot_row(ra, Cfg::SA) + qa : 2 * kMmKB * Cfg::SA + slot_row(rb, Cfg::SB) + qb);
#pragma unroll
    for (int u = 0; u < (ROOTS ? UC : 0); ++u)
      *reinterpret_cast<double2*>(st + (COS_A ? (RA / 2) * Cfg::SA : 4 * Cfg::SB) * u) = cosv[u];
  };
  auto start = [&](unsigned tile) {  // the tile's coordinates and first copies
    const unsigned rest = tile / p.nm;
    m0n = (int)(tile - rest * p.nm) * Cfg::MT;
    btn = rest / p.nn;
    n0n = (int)(rest - btn * p.nn) * kMmNT;
    pa = p.A + (int64_t)btn * p.bA + (int64_t)ra * p.lda + m0n + qa;
    pb = p.B + (int64_t)btn * p.bB + (int64_t)rb * p.ldb + n0n + qb;
    ka = m0n + qa < p.wa ? p.K - ra : 0;
    kb_ = n0n + qb < p.wb ? p.K - rb : 0;
#pragma unroll
    for (int s = 0; s < kMmStages - 1; ++s) {
      if (s < nk) {
        load(s, s);
        form(s);
        put(s);
      }
      asm volatile("cp.async.commit_group;\n" ::: "memory");
    }
  };
  if (blockIdx.x < total) start(blockIdx.x);

  for (unsigned tile = blockIdx.x; tile < total; tile += gridDim.x) {
    const int m0 = m0n, n0 = n0n;
    const unsigned bt = btn;
    double acc[2][MW][2][2];
#pragma unroll
    for (int e = 0; e < 2; ++e)
#pragma unroll
      for (int i = 0; i < MW; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) acc[e][i][j][0] = acc[e][i][j][1] = 0.0;
    // groups of 16 rows (two accumulator rows) this warp computes: group I holds
    // rows m0 + 16 (2 I + wm); none where the warp's columns lie beyond N
    const int mg = (p.M - m0 + 15) / 16;
    const int mw = n0 + 16 * wn >= p.N ? 0 : mg > wm ? (mg - wm + 1) / 2 : 0;
    // GW: groups computed, a compile-time count (a predicated-off mma still
    // takes its slot of the tensor pipe)
    auto loop = [&](auto gw) {
      constexpr int GW = decltype(gw)::value;
      for (int kb = 0; kb < nk; ++kb) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(kMmStages - 2) : "memory");
        __syncthreads();
        const bool more = kb + kMmStages - 1 < nk;
        if (more) {
          load(kb + kMmStages - 1, (kb + kMmStages - 1) % kMmStages);
          form(kb + kMmStages - 1);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        if constexpr (GW > 0) {
          const double* as = mm_sm + (kb % kMmStages) * Cfg::STAGE;
          const double* bs = as + 2 * kMmKB * Cfg::SA;
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const double* ar = as + (e * kMmKB + t) * Cfg::SA + 16 * wm + g;
            const double* br = bs + (e * kMmKB + t) * Cfg::SB + 16 * wn + g;
            const double b00 = br[0], b01 = br[4 * Cfg::SB], b10 = br[8], b11 = br[4 * Cfg::SB + 8];
#pragma unroll
            for (int i = 0; i < GW; ++i) {
              const double a[4] = {ar[32 * i], ar[32 * i + 8], ar[4 * Cfg::SA + 32 * i], ar[4 * Cfg::SA + 32 * i + 8]};
              dmma(acc[e][2 * i][0], acc[e][2 * i + 1][0], a, b00, b01);
              dmma(acc[e][2 * i][1], acc[e][2 * i + 1][1], a, b10, b11);
            }
          }
        }
        if (more) put((kb + kMmStages - 1) % kMmStages);
      }
    };
    if (mw == 0) loop(std::integral_constant<int, 0>());
    else if (mw < MW / 2) loop(std::integral_constant<int, 1>());
    else loop(std::integral_constant<int, MW / 2>());
    __syncthreads();  // every warp has read the last stage
    if (tile + gridDim.x < total) start(tile + gridDim.x);

    // ---- output: accumulator row i holds row m = m0 + 16 (2 (i / 2) + wm) +
    //      8 (i % 2) + g, columns n0 + 16 wn + 8 j + 2 t + {0, 1} ----
    if constexpr (OUT == MM_FOLD_M) {
      double* D = p.D + (int64_t)bt * p.bD;
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int n = n0 + 16 * wn + 8 * j + 2 * t;
        if (n >= p.N) continue;  // rows are even: both columns exist
#pragma unroll
        for (int i = 0; i < MW; ++i) {
          const int m = m0 + 16 * (2 * (i / 2) + wm) + 8 * (i % 2) + g;
          if (m >= p.M) continue;
          const double e0 = acc[0][i][j][0], e1 = acc[0][i][j][1], o0 = acc[1][i][j][0], o1 = acc[1][i][j][1];
          *reinterpret_cast<double2*>(D + (int64_t)m * p.ldd + n) = make_double2(e0 + o0, e1 + o1);
          if (2 * m + 1 != p.Nfull)
            *reinterpret_cast<double2*>(D + (int64_t)(p.Nfull - 1 - m) * p.ldd + n) = make_double2(e0 - o0, e1 - o1);
        }
      }
    } else {
      // y_n, then y_{N-1-n}, through shared memory: lanes on consecutive columns
      double* so = mm_sm + Cfg::OFF_OUT;
      const int col = tid & 63, r0 = tid >> 6, n = n0 + col;
#pragma unroll 1
      for (int half = 0; half < 2; ++half) {
        if (half) __syncthreads();
        const double sg = half ? -1.0 : 1.0;
#pragma unroll
        for (int i = 0; i < MW; ++i)
#pragma unroll
          for (int j = 0; j < 2; ++j)
            *reinterpret_cast<double2*>(so + (16 * (2 * (i / 2) + wm) + 8 * (i % 2) + g) * Cfg::SO + 16 * wn + 8 * j +
                                        2 * t) = make_double2(fma(sg, acc[1][i][j][0], acc[0][i][j][0]),
                                                              fma(sg, acc[1][i][j][1], acc[0][i][j][1]));
        __syncthreads();
        if (n >= p.N) continue;
        if constexpr (OUT == MM_FOLD_N) {
          if (half && 2 * n + 1 == p.Nfull) continue;
          double* D = p.D + (int64_t)bt * p.bD + (half ? p.Nfull - 1 - n : n);
#pragma unroll 4
          for (int r = r0; r < Cfg::MT; r += 4)
            if (m0 + r < p.M) D[(int64_t)(m0 + r) * p.ldd] = so[r * Cfg::SO + col];
        } else {
          const Epilogue& e = p.epi;
          const int y = n / p.n0p, x = n - y * p.n0p;
          if (x >= p.n0) continue;
          const bool blend = e.mode != 0;
          const int64_t zs = blend ? e.L[0] * e.L[1] : (int64_t)p.n0 * p.n1;
          const int64_t base = blend ? e.off[0] + x + e.L[0] * (e.off[1] + y + e.L[1] * e.off[2]) : x + (int64_t)p.n0 * y;
          // rows z = z0 + dz r, r < rows (the middle row of an odd length once)
          const int z0 = half ? p.Nfull - 1 - m0 : m0, dz = half ? -1 : 1;
          const int rows = min(Cfg::MT, (half ? p.Nfull / 2 : p.M) - m0);
          double* o = static_cast<double*>(e.out) + (int64_t)bt * p.bD + base + zs * (z0 + dz * r0);
          const int64_t step = 4 * dz * zs;
          const double ms = e.marginal ? e.ms : 1.0, mu = e.marginal ? e.mmu : 0.0;
          const double* sr = so + r0 * Cfg::SO + col;
          if (!blend) {
#pragma unroll 4
            for (int r = r0; r < rows; r += 4, o += step, sr += 4 * Cfg::SO) {
              const double w = sr[0];
              *o = EXP ? exp(w * ms + mu) : w * ms + mu;
            }
            continue;
          }
          const uint8_t fxy = e.ax[1].flags[y] & e.ax[0].flags[x];
          if (!(fxy & 1)) continue;
          const double sxy = e.apply_pou ? e.ax[1].sw64[y] * e.ax[0].sw64[x] : 1.0;
          const uint8_t* fz = e.ax[2].flags + z0 + dz * r0;
          const double* sz = e.ax[2].sw64 + z0 + dz * r0;
#pragma unroll 1
          for (int r = r0; r < rows; r += 16) {  // four rows: their reads before their writes
            double w[4], old[4];
            uint8_t f[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              f[u] = r + 4 * u < rows ? (uint8_t)(fxy & fz[4 * dz * u]) : (uint8_t)0;
              old[u] = (f[u] & 3) == 1 ? o[step * u] : 0.0;
              w[u] = sr[4 * u * Cfg::SO];
              if (e.apply_pou && (f[u] & 1)) w[u] = w[u] * (sxy * sz[4 * dz * u]);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              if (!(f[u] & 1)) continue;
              if (!(f[u] & 2)) w[u] = old[u] + w[u];
              if (f[u] & 4) {
                w[u] = w[u] * ms + mu;
                if constexpr (EXP) w[u] = exp(w[u]);
              }
              o[step * u] = w[u];
            }
            o += 4 * step;
            sr += 16 * Cfg::SO;
            fz += 16 * dz;
            sz += 16 * dz;
          }
        }
      }
    }
  }
}

template <int MW, int OUT, bool ROOTS> static cudaError_t run_mm_w(DctMM p, int64_t batch, cudaStream_t s) {
  using Cfg = MmCfg<MW>;
  p.nm = (p.M + Cfg::MT - 1) / Cfg::MT;
  p.nn = (p.N + kMmNT - 1) / kMmNT;
  const int64_t tiles = (int64_t)p.nm * p.nn * batch;
  if (tiles < 1 || tiles > 2147483647LL) return cudaErrorInvalidValue;
  p.batch = (int)batch;
  p.inv = ~(uint64_t)0 / (4 * (uint64_t)p.Nfull);
  const cudaError_t e = cudaFuncSetAttribute(k_dct_mm<MW, OUT, ROOTS>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM);
  if (e != cudaSuccess) return e;
  k_dct_mm<MW, OUT, ROOTS><<<(unsigned)std::min<int64_t>(tiles, 2 * 148), 256, Cfg::SMEM, s>>>(p);
  return cudaGetLastError();
}
// Tiles of 64 rows reuse a B fragment most; 32 only where M is that small.
template <int OUT, bool ROOTS> static cudaError_t run_mm_r(const DctMM& p, int64_t batch, cudaStream_t s) {
  if (p.M <= 32) return run_mm_w<2, OUT, ROOTS>(p, batch, s);
  return run_mm_w<4, OUT, ROOTS>(p, batch, s);
}
template <int OUT> static cudaError_t run_mm(const DctMM& p, int64_t batch, cudaStream_t s) {
  return p.ctab ? run_mm_r<OUT, true>(p, batch, s) : run_mm_r<OUT, false>(p, batch, s);
}

void dct_sizes(const int Np[3], const int K[3], int64_t* sk, int64_t* t1, int64_t* t2) {
  const int64_t lp = ((int64_t)K[1] * K[2] + 1) / 2 * 2, n0p = (Np[0] + 1) / 2 * 2;
  *sk = K[0] * lp;
  *t1 = (int64_t)K[1] * K[2] * n0p;
  *t2 = (int64_t)K[2] * Np[1] * n0p;
}

cudaError_t launch_dct_literal(const DctArgs& a_in, cudaStream_t s) {
  DctArgs a = a_in;
  const int N0 = a.Np[0], N1 = a.Np[1], N2 = a.Np[2], K0 = a.K[0], K1 = a.K[1], K2 = a.K[2];
  const int n0p = (N0 + 1) / 2 * 2;
  const int H[3] = {(N0 + 1) / 2, (N1 + 1) / 2, (N2 + 1) / 2};
  const int hp[3] = {(H[0] + 1) / 2 * 2, (H[1] + 1) / 2 * 2, (H[2] + 1) / 2 * 2};
  int64_t nsk, n1, n2;
  dct_sizes(a.Np, a.K, &nsk, &n1, &n2);
  if ((int64_t)N1 * n0p > 2147483647LL - 64 || (int64_t)K1 * K2 > 2147483647LL - 64) return cudaErrorInvalidValue;
  a.lp = ((int64_t)K1 * K2 + 1) / 2 * 2;
  k_dct_spec<<<dim3((unsigned)((K1 * K2 + 127) / 128), std::min(K0, 65535), a.nt), 128, 0, s>>>(a);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  DctMM p{};
  // x: rows (j, k) of the octant
  p.A = a.sk; p.lda = a.lp; p.wa = (int)a.lp; p.bA = nsk;
  p.ctab = a.roots[0];
  p.B = a.tab[0]; p.ldb = hp[0]; p.wb = hp[0]; p.bB = 0;
  p.D = a.t1; p.ldd = n0p; p.bD = n1;
  p.M = K1 * K2; p.N = H[0]; p.K = K0; p.Nfull = N0;
  if ((e = run_mm<MM_FOLD_N>(p, a.nt, s)) != cudaSuccess) return e;
  // y: per kz (and tile), rows of x
  p.ctab = a.roots[1];
  p.A = a.tab[1]; p.lda = hp[1]; p.wa = hp[1]; p.bA = 0;
  p.B = a.t1; p.ldb = n0p; p.wb = n0p; p.bB = (int64_t)K1 * n0p;
  p.D = a.t2; p.ldd = n0p; p.bD = (int64_t)N1 * n0p;
  p.M = H[1]; p.N = n0p; p.K = K1; p.Nfull = N1;
  if ((e = run_mm<MM_FOLD_M>(p, (int64_t)K2 * a.nt, s)) != cudaSuccess) return e;
  // z: whole planes, through the output stage
  p.ctab = a.roots[2];
  p.A = a.tab[2]; p.lda = hp[2]; p.wa = hp[2]; p.bA = 0;
  p.B = a.t2; p.ldb = N1 * n0p; p.wb = N1 * n0p; p.bB = n2;
  p.D = nullptr; p.ldd = 0; p.bD = (int64_t)N0 * N1 * N2;
  p.M = H[2]; p.N = N1 * n0p; p.K = K2; p.Nfull = N2;
  p.n0 = N0; p.n0p = n0p; p.n1 = N1;
  p.epi = a.epi;
  return a.epi.marginal == 2 ? run_mm<MM_FINAL_EXP>(p, a.nt, s) : run_mm<MM_FINAL>(p, a.nt, s);
}

// Blended field from tiles held in memory, one thread a point: the tiles that
// cover it (at most two along each axis) summed in rank order, the order in
// which one tile after another would add to it.
__global__ void __launch_bounds__(256) k_blend_gather(const BlendGather g) {
  const int64_t n = g.L[0] * g.L[1] * g.L[2];
  const int64_t nt = (int64_t)g.Np[0] * g.Np[1] * g.Np[2];
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t q = i / g.L[0];
    const int X[3] = {(int)(i - q * g.L[0]), (int)(q % g.L[1]), (int)(q / g.L[1])};
    int lo[3], hi[3];  // tile positions along each axis
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const int st = g.Np[d] - g.No[d];
      if (g.T[d] == 1 || st <= 0) {
        lo[d] = 0;
        hi[d] = g.T[d] - 1;
      } else {
        hi[d] = min(X[d] / st, g.T[d] - 1);
        lo[d] = X[d] >= g.Np[d] ? (X[d] - g.Np[d]) / st + 1 : 0;
      }
    }
    double acc = 0.0;
    bool first = true;
    for (int tz = lo[2]; tz <= hi[2]; ++tz)
      for (int ty = lo[1]; ty <= hi[1]; ++ty)
        for (int tx = lo[0]; tx <= hi[0]; ++tx) {
          const int t[3] = {tx, ty, tz};
          int c[3];
          uint8_t f = 7;
          double s[3];
#pragma unroll
          for (int d = 0; d < 3; ++d) {
            c[d] = X[d] - t[d] * (g.Np[d] - g.No[d]);
            const int64_t rk = (d == 0 ? 1 : d == 1 ? g.T[0] : g.T[0] * g.T[1]) * (int64_t)t[d];
            f &= g.fl[d][rk * g.fls + c[d]];
            s[d] = g.pou ? g.sw[d][rk * g.sws + c[d]] : 1.0;
          }
          if (!(f & 1)) continue;
          const int64_t r = tx + (int64_t)g.T[0] * (ty + (int64_t)g.T[1] * tz);
          double v = g.tiles[r * nt + c[0] + (int64_t)g.Np[0] * (c[1] + (int64_t)g.Np[1] * c[2])];
          if (g.pou) v = v * (s[1] * s[2] * s[0]);
          acc = first || (f & 2) ? v : acc + v;
          first = false;
        }
    if (g.marginal == 1) acc = acc * g.ms + g.mu;
    else if (g.marginal == 2) acc = exp(acc * g.ms + g.mu);
    g.out[i] = acc;
  }
}

cudaError_t launch_blend_gather(const BlendGather& g, cudaStream_t s) {
  const int64_t n = g.L[0] * g.L[1] * g.L[2];
  k_blend_gather<<<(unsigned)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, 148 * 32)), 256, 0, s>>>(g);
  return cudaGetLastError();
}

}  // namespace scarl
