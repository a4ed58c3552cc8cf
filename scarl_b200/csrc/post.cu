// post.cu -- standalone post steps of the localization method, each a
// memory-bound elementwise or gather pass over HBM:
//   k_apply_pou    : apply_UnityPartition_mtx (SRC_F/main_ScaRL.f90:1216-1301);
//   k_add_overlap  : add_overlap over all tiles held in HBM (:984-1210);
//   k_marginal     : multiVariateTransformation (:1355-1395);
//   k_affine       : (x - a) / b, the standardisation of normalize_field (:903-953);
//   k_sums         : FP64 sums of x and x^2 per realisation (moments, normalisation).
#include <algorithm>

#include "epilogue.cuh"
#include "scarl_internal.h"

namespace scarl {

static inline unsigned grid_for(int64_t n, int threads, int cap = 148 * 32) {
  int64_t g = (n + threads - 1) / threads;
  return (unsigned)std::max<int64_t>(1, std::min<int64_t>(g, cap));
}

struct PouAxes { BlendAxis ax[3]; };

// A warp a row of x (the row's y and z found once, with 32-bit arithmetic where
// the rows and the walk's last step allow it: I): f *= sqrt(w), the factors
// multiplied in the reference's order.  A factor of exactly 1, the inside of the
// tile, leaves the value as it is: neither read nor written.  Bound by launch
// latency at the sizes of the drop-in steps (95 x 78 x 83 FP64 points: 12.8 -> 11.4
// us between two timing events, of which an empty kernel takes about 5), against a
// thread a point with 64-bit divisions.
constexpr int kRowsPerBlock = 8, kRowBlocks = 148 * 64;
template <typename T, typename I>
__global__ void __launch_bounds__(32 * kRowsPerBlock) k_apply_pou(T* __restrict__ f, int Nx, int Ny, I nrows,
                                                                  const PouAxes p) {
  const int lane = threadIdx.x & 31;
  for (I row = (I)(blockIdx.x * kRowsPerBlock + (threadIdx.x >> 5)); row < nrows; row += (I)(gridDim.x * kRowsPerBlock)) {
    const int z = (int)(row / Ny), y = (int)(row - (I)z * Ny);
    const double ly = p.ax[1].lo[y], lz = p.ax[2].lo[z], hy = p.ax[1].hi[y], hz = p.ax[2].hi[z];
    T* r = f + (int64_t)row * Nx;
    for (unsigned x = lane; x < (unsigned)Nx; x += 32) {
      double w = p.ax[0].lo[x];
      w = __dmul_rn(w, ly);
      w = __dmul_rn(w, lz);
      w = __dmul_rn(w, p.ax[0].hi[x]);
      w = __dmul_rn(w, hy);
      w = __dmul_rn(w, hz);
      if (w != 1.0) r[x] = (T)((double)r[x] * sqrt(w));
    }
  }
}

template <typename T>
static void apply_pou(unsigned g, T* field, const int Np[3], int64_t rows, const PouAxes& p, cudaStream_t s) {
  if (rows <= 2147483647LL - kRowBlocks * kRowsPerBlock)
    k_apply_pou<T, int><<<g, 32 * kRowsPerBlock, 0, s>>>(field, Np[0], Np[1], (int)rows, p);
  else
    k_apply_pou<T, int64_t><<<g, 32 * kRowsPerBlock, 0, s>>>(field, Np[0], Np[1], rows, p);
}

cudaError_t launch_apply_pou(int dt, void* field, const int Np[3], const BlendAxis ax[3],
                             cudaStream_t s) {
  PouAxes p{{ax[0], ax[1], ax[2]}};
  const int64_t rows = (int64_t)Np[1] * Np[2];
  const unsigned g = grid_for(rows, kRowsPerBlock, kRowBlocks);
  if (dt == 8) apply_pou(g, (double*)field, Np, rows, p, s);
  else apply_pou(g, (float*)field, Np, rows, p, s);
  return cudaGetLastError();
}

// out[r] = in[r] + sum over the 26 directions s (reference order, x fastest)
// of in[r - s] on the receiver's region(-s), read at the sender's region(s).
// out holds in's values already: points that no other tile covers are left.
// A warp a row of x: which (y, z) directions reach the row is found once per
// row, which x directions by two compares a point.  8 tiles of 95 x 78 x 83:
// 138 -> 33 us between timing events, against a thread a point that tested
// every direction.
struct OvlArgs { int Np[3], No[3], T[3]; };

__global__ void __launch_bounds__(32 * kRowsPerBlock) k_add_overlap(const double* __restrict__ in, double* __restrict__ out,
                                                                    const OvlArgs a, int64_t nrows) {
  const int lane = threadIdx.x & 31;
  const int Nx = a.Np[0], Ny = a.Np[1], Nz = a.Np[2];
  const int64_t rows = (int64_t)Ny * Nz;
  // direction s along axis d reaches coordinate c of a tile at position pos:
  // s = 1 the low side, -1 the high side, 0 the tile's own extent; degenerate
  // regions (one point) never
  auto reaches = [&](int d, int s, int c, int pos) -> bool {
    if (s == 0) return a.Np[d] > 1;
    if (a.No[d] < 2) return false;
    return s == 1 ? pos > 0 && c < a.No[d] : pos < a.T[d] - 1 && c >= a.Np[d] - a.No[d];
  };
  for (int64_t q = (int64_t)blockIdx.x * kRowsPerBlock + (threadIdx.x >> 5); q < nrows;
       q += (int64_t)gridDim.x * kRowsPerBlock) {
    const int r = (int)(q / rows);
    const int64_t yz = q - r * rows;
    const int z = (int)(yz / Ny), y = (int)(yz - (int64_t)z * Ny);
    const int pz = r / (a.T[0] * a.T[1]), rest = r - pz * a.T[0] * a.T[1], py = rest / a.T[0], px = rest - py * a.T[0];
    unsigned m = 0;  // bit 3 (kk + 1) + (jj + 1)
    for (int kk = -1; kk <= 1; ++kk)
      for (int jj = -1; jj <= 1; ++jj)
        if (reaches(2, kk, z, pz) && reaches(1, jj, y, py)) m |= 1u << (3 * (kk + 1) + jj + 1);
    if (!m) continue;
    const int dx = Nx - a.No[0], dy = Ny - a.No[1], dz = Nz - a.No[2];
    for (int64_t x = lane; x < Nx; x += 32) {
      const bool xl = reaches(0, 1, x, px), xh = reaches(0, -1, x, px), x0 = Nx > 1;
      if (!xl && !xh && (m & ~(1u << 4)) == 0) continue;
      if (!xl && !xh && !x0) continue;
      double acc = 0.0;
      for (unsigned left = m; left; left &= left - 1) {
        const int b = __ffs(left) - 1, kk = b / 3 - 1, jj = b - 3 * (kk + 1) - 1;
        const int rs = r - a.T[0] * (a.T[1] * kk + jj);
        const double* src = in + ((int64_t)rs * rows + (int64_t)(z + kk * dz) * Ny + (y + jj * dy)) * Nx;
        const int64_t tile = (int64_t)rows * Nx;
        if (xh) acc = acc + src[tile + x - dx];           // ii = -1: the next tile along x
        if (x0 && b != 4) acc = acc + src[x];             // ii = 0
        if (xl) acc = acc + src[x + dx - tile];           // ii = 1: the previous one
      }
      const int64_t i = q * Nx + x;
      out[i] = in[i] + acc;
    }
  }
}

cudaError_t launch_add_overlap(const double* in, double* out, const int Np[3],
                               const int Np_ovlp[3], const int topo[3], cudaStream_t s) {
  OvlArgs a;
  for (int d = 0; d < 3; ++d) { a.Np[d] = Np[d]; a.No[d] = Np_ovlp[d]; a.T[d] = topo[d]; }
  const int64_t rows = (int64_t)Np[1] * Np[2] * topo[0] * topo[1] * topo[2];
  k_add_overlap<<<grid_for(rows, kRowsPerBlock, kRowBlocks), 32 * kRowsPerBlock, 0, s>>>(in, out, a, rows);
  return cudaGetLastError();
}

template <typename T>
__global__ void k_marginal(T* __restrict__ f, int64_t n, int kind, T sc, T mu) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    T v = f[i] * sc + mu;
    f[i] = (kind == 2) ? exp(v) : v;
  }
}

cudaError_t launch_marginal(int dt, void* f, int64_t n, int kind, double sc, double mu,
                            cudaStream_t s) {
  if (dt == 8) k_marginal<double><<<grid_for(n, 256), 256, 0, s>>>((double*)f, n, kind, sc, mu);
  else k_marginal<float><<<grid_for(n, 256), 256, 0, s>>>((float*)f, n, kind, (float)sc, (float)mu);
  return cudaGetLastError();
}

template <typename T>
__global__ void k_affine(T* __restrict__ f, int64_t n, T sub, T div) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    f[i] = (f[i] - sub) / div;
}

cudaError_t launch_affine(int dt, void* f, int64_t n, double sub, double div, cudaStream_t s) {
  if (dt == 8) k_affine<double><<<grid_for(n, 256), 256, 0, s>>>((double*)f, n, sub, div);
  else k_affine<float><<<grid_for(n, 256), 256, 0, s>>>((float*)f, n, (float)sub, (float)div);
  return cudaGetLastError();
}

// Deterministic FP64 partial sums: block (b, e) covers a fixed slice of
// realisation e; partial[(e*nb + b)*2 + {0,1}] = {sum x, sum x^2}.
constexpr int kSumT = 256;
int sums_blocks(int64_t xN) { return (int)std::max<int64_t>(1, std::min<int64_t>((xN + 4095) / 4096, 148 * 4)); }

template <typename T>
__global__ void __launch_bounds__(kSumT) k_sums(const T* __restrict__ f, int64_t xN, double* partial) {
  const int e = blockIdx.y, nb = gridDim.x;
  const T* p = f + (int64_t)e * xN;
  const int64_t chunk = (xN + nb - 1) / nb;
  const int64_t lo = (int64_t)blockIdx.x * chunk, hi = (lo + chunk < xN) ? lo + chunk : xN;
  double s = 0.0, s2 = 0.0;
  constexpr int U = 8;  // independent loads in flight per thread
  int64_t i = lo + threadIdx.x;
  for (; i + (U - 1) * kSumT < hi; i += U * kSumT) {
    T v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) v[u] = __ldg(p + i + u * kSumT);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const double d = (double)v[u];
      s += d;
      s2 += d * d;
    }
  }
  for (; i < hi; i += kSumT) {
    const double v = (double)p[i];
    s += v;
    s2 += v * v;
  }
  __shared__ double r1[kSumT / 32], r2[kSumT / 32];
  for (int o = 16; o > 0; o >>= 1) {
    s += __shfl_down_sync(0xffffffffu, s, o);
    s2 += __shfl_down_sync(0xffffffffu, s2, o);
  }
  if ((threadIdx.x & 31) == 0) { r1[threadIdx.x >> 5] = s; r2[threadIdx.x >> 5] = s2; }
  __syncthreads();
  if (threadIdx.x < 32) {
    s = threadIdx.x < kSumT / 32 ? r1[threadIdx.x] : 0.0;
    s2 = threadIdx.x < kSumT / 32 ? r2[threadIdx.x] : 0.0;
    for (int o = 16; o > 0; o >>= 1) {
      s += __shfl_down_sync(0xffffffffu, s, o);
      s2 += __shfl_down_sync(0xffffffffu, s2, o);
    }
    if (threadIdx.x == 0) {
      partial[((int64_t)e * nb + blockIdx.x) * 2] = s;
      partial[((int64_t)e * nb + blockIdx.x) * 2 + 1] = s2;
    }
  }
}

cudaError_t launch_sums(int dt, const void* f, int64_t xN, int nmc, double* partial, int nb,
                        cudaStream_t s) {
  dim3 grid(nb, nmc);
  if (dt == 8) k_sums<double><<<grid, kSumT, 0, s>>>((const double*)f, xN, partial);
  else k_sums<float><<<grid, kSumT, 0, s>>>((const float*)f, xN, partial);
  return cudaGetLastError();
}

}  // namespace scarl
