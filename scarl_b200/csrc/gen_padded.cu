// gen_padded.cu -- dispatch of the padded periodic-grid generator passes
// (kernels in gen_kernels.cuh, variants in gen_launch.cuh, instantiated per
// precision and line length by gen_inst.cu) and the FP64 spectral
// normalisation sum.
#include "gen_launch.cuh"

namespace scarl {

// Defined and explicitly instantiated in gen_inst.cu.
template <typename T, int N>
cudaError_t run_pass_len(int pass, int v, const GenArgs& a, const BatchMap* bm, int* nb,
                         cudaStream_t s);

template <typename T>
static cudaError_t run_pass_t(int pass, int v, const GenArgs& a, const BatchMap* bm, int* nb,
                              cudaStream_t s) {
  const int N = pass == 1 ? a.P[2] : (pass == 2 ? a.P[1] : a.P[0] / 2);
  switch (N) {
    case 4: return run_pass_len<T, 4>(pass, v, a, bm, nb, s);
    case 8: return run_pass_len<T, 8>(pass, v, a, bm, nb, s);
    case 16: return run_pass_len<T, 16>(pass, v, a, bm, nb, s);
    case 24: return run_pass_len<T, 24>(pass, v, a, bm, nb, s);
    case 32: return run_pass_len<T, 32>(pass, v, a, bm, nb, s);
    case 40: return run_pass_len<T, 40>(pass, v, a, bm, nb, s);
    case 48: return run_pass_len<T, 48>(pass, v, a, bm, nb, s);
    case 56: return run_pass_len<T, 56>(pass, v, a, bm, nb, s);
    case 64: return run_pass_len<T, 64>(pass, v, a, bm, nb, s);
    case 80: return run_pass_len<T, 80>(pass, v, a, bm, nb, s);
    case 96: return run_pass_len<T, 96>(pass, v, a, bm, nb, s);
    case 112: return run_pass_len<T, 112>(pass, v, a, bm, nb, s);
    case 128: return run_pass_len<T, 128>(pass, v, a, bm, nb, s);
    case 160: return run_pass_len<T, 160>(pass, v, a, bm, nb, s);
    case 192: return run_pass_len<T, 192>(pass, v, a, bm, nb, s);
    case 224: return run_pass_len<T, 224>(pass, v, a, bm, nb, s);
    case 256: return run_pass_len<T, 256>(pass, v, a, bm, nb, s);
    case 320: return run_pass_len<T, 320>(pass, v, a, bm, nb, s);
    case 384: return run_pass_len<T, 384>(pass, v, a, bm, nb, s);
    case 448: return run_pass_len<T, 448>(pass, v, a, bm, nb, s);
    case 512: return run_pass_len<T, 512>(pass, v, a, bm, nb, s);
    case 640: return run_pass_len<T, 640>(pass, v, a, bm, nb, s);
    case 768: return run_pass_len<T, 768>(pass, v, a, bm, nb, s);
    case 896: return run_pass_len<T, 896>(pass, v, a, bm, nb, s);
    case 1024: return run_pass_len<T, 1024>(pass, v, a, bm, nb, s);
    case 1280: return run_pass_len<T, 1280>(pass, v, a, bm, nb, s);
    case 1536: return run_pass_len<T, 1536>(pass, v, a, bm, nb, s);
    case 1792: return run_pass_len<T, 1792>(pass, v, a, bm, nb, s);
    case 2048: return run_pass_len<T, 2048>(pass, v, a, bm, nb, s);
    default: return cudaErrorInvalidValue;
  }
}

static cudaError_t run_pass_dt(int dt, int pass, int v, const GenArgs& a, const BatchMap* bm,
                               int* nb, cudaStream_t s) {
  if (pass < 1 || pass > 3) return cudaErrorInvalidValue;
  return dt == 8 ? run_pass_t<double>(pass, v, a, bm, nb, s)
                 : run_pass_t<float>(pass, v, a, bm, nb, s);
}

void philox_schedule(GenArgs* a) {
  for (int r = 0; r < 10; ++r) {
    a->ks[r] = a->k0 + (uint32_t)r * 0x9E3779B9u;
    a->ks[10 + r] = a->k1 + (uint32_t)r * 0xBB67AE85u;
  }
}

cudaError_t launch_gen_pass(int dt, int pass, const GenArgs& a_in, cudaStream_t s) {
  if (pass < 1 || pass > 3) return cudaErrorInvalidValue;
  GenArgs a = a_in;
  philox_schedule(&a);
  if (pass == 1 && a.split && dt == 4 && a.spec == SPEC_PHILOX && gen_z_tc_supported(a.P[2]))
    return launch_gen_z_tc(a, s);
  if (pass == 3 && c2r_x_tc_used(dt, a)) return launch_c2r_x_tc(a, s);
  // injected and literal spectra run the first pass-1 variant only
  return run_pass_dt(dt, pass, pass == 1 && a.spec != SPEC_PHILOX ? 0 : a.var[pass - 1], a, nullptr, nullptr, s);
}

cudaError_t launch_gen_pass_batch(int dt, int pass, int v, const GenArgs& rep, const BatchMap& m,
                                  cudaStream_t s) {
  if (m.n < 1 || m.total < 1) return cudaErrorInvalidValue;
  return run_pass_dt(dt, pass, v, rep, &m, nullptr, s);
}

int gen_pass_blocks(int dt, int pass, int v, const GenArgs& a) {
  int nb = 0;
  if (run_pass_dt(dt, pass, v, a, nullptr, &nb, nullptr) != cudaSuccess) return -1;
  return nb;
}

// Every pass-3 kernel stores one moment pair a block.
int gen_pass3_partials(int dt, int v, const GenArgs& a) {
  if (c2r_x_tc_used(dt, a)) return c2r_x_tc_blocks(a);
  return gen_pass_blocks(dt, 3, v, a);
}

// The variant an untuned (precision, pass, length) runs: the fastest of a sweep
// of every variant over lengths 32 .. 2048 on grids of 12 - 24 M modes, crop mode.
//
// Passes 1 and 2: the two-stage kernels for lengths m 2^a (m = 3, 5, 7), whose
// engine plans take four or five stages (FP32 pass 1 / pass 2, us: 224 71 / 25
// against 89 / 33, 384 66 / 23 against 70 / 31, 448 82 / 29 against 91 / 35; FP64
// 224 92 / 27 against 127 / 33), and for short powers of two.  Longer powers of two
// keep two or three engine stages, with 32 values a thread in the FP32 pass 2 from
// 512 on (31.8 against 35.4, 1024 36.9 against 45.6) and eight in the FP64 pass 1
// (256 94.5 against 98.7, 1024 118 against 140).
// Pass 3: the two-stage kernel where it serves the half length (FP32 224 / 256 /
// 384 / 512: 47 / 45 / 48 / 65 against 58 / 62 / 66 / 72 for the best other; FP64
// 112 / 224 / 256: 46 / 45 / 46 against 80 / 117 / 72), except FP32 lines of 64 and
// 128 (two engine stages, no staging of the outputs: 53.5 against 59.7 and 51.6
// against 61.3).
int gen_default_variant(int dt, int pass, const GenArgs& a) {
  const bool f32 = dt == 4;
  if (pass == 3) {
    const int N = a.P[0] / 2;
    if (f32 && N == 64) return 3;
    if (f32 && N == 128) return 0;
    const int v = f32 ? kTwoRow<float> : kTwoRow<double>;
    return gen_pass_blocks(dt, pass, v, a) > 0 ? v : 0;
  }
  const int N = a.P[pass == 1 ? 2 : 1], two = f32 ? kTwoCol<float> : kTwoCol<double>;
  const bool mixed = (N & (N - 1)) != 0;
  if ((mixed || N <= (pass == 1 ? (f32 ? 256 : 64) : (f32 ? 32 : 64))) && gen_pass_blocks(dt, pass, two, a) > 0)
    return two;
  if (f32) {
    if (pass == 1) return N >= 1024 ? 1 : 0;
    return mixed ? (N > 1024 ? 1 : 0) : N >= 1024 ? 3 : N >= 512 ? 4 : 0;
  }
  return pass == 1 && !mixed && N >= 128 ? 2 : 0;
}

int gen_variant_count(int dt, int pass) {
  if (pass == 3) return dt == 8 ? RowVars<double>::n : RowVars<float>::n + kShflVars<float>;
  if (pass == 2 && dt == 4) return ColVars<float>::n + kDirectVars<float>;
  return dt == 8 ? ColVars<double>::n : ColVars<float>::n;
}

// ---------------------------------------------------------------------------
// FP64 spectral variance-normalisation sum over the full periodic grid.
// ---------------------------------------------------------------------------
constexpr int kSumThreads = 256;
int spectrum_sum_blocks() { return 148 * 8; }

__global__ void __launch_bounds__(kSumThreads) k_spec_sum(const GenArgs a, const double* rx,
                                                          const double* ry, const double* rz,
                                                          double craw2, double* partial) {
  const double* qx = static_cast<const double*>(a.qx);
  const double* qy = static_cast<const double*>(a.qy);
  const double* qz = static_cast<const double*>(a.qz);
  const int64_t total = (int64_t)a.Hx * a.P[1] * a.P[2];
  double acc = 0.0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int kx = (int)(i % a.Hx);
    const int64_t r = i / a.Hx;
    const int ky = (int)(r % a.P[1]);
    const int kz = (int)(r / a.P[1]);
    const double c = (kx == 0 || 2 * kx == a.P[0]) ? 1.0 : 2.0;
    double v;
    if (a.amp == AMP_SEPARABLE) {
      const double A = rx[kx] * ry[ky] * rz[kz];
      v = A * A;
    } else {
      v = craw2 * pow(1.0 + qx[kx] + qy[ky] + qz[kz], 2.0 * a.expo);
    }
    acc += c * v;
  }
  __shared__ double red[kSumThreads / 32];
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x < 32) {
    double v = threadIdx.x < kSumThreads / 32 ? red[threadIdx.x] : 0.0;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (threadIdx.x == 0) partial[blockIdx.x] = v;
  }
}

cudaError_t launch_spectrum_sum(const GenArgs& a, const double* rx, const double* ry,
                                const double* rz, double craw2, double* partial, int nblocks,
                                cudaStream_t s) {
  k_spec_sum<<<nblocks, kSumThreads, 0, s>>>(a, rx, ry, rz, craw2, partial);
  return cudaGetLastError();
}

}  // namespace scarl
