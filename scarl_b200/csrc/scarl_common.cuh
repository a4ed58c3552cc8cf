// scarl_common.cuh -- device-side helpers shared by every scarl_b200 kernel:
// complex arithmetic on float2/double2, the Philox4x32-10 counter RNG, the
// Park-Miller jump-ahead, and the exact radix-32 unit-root constants.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace scarl {

template <typename T> struct cplx_of;
template <> struct cplx_of<float> { using type = float2; };
template <> struct cplx_of<double> { using type = double2; };
template <typename T> using cplx_t = typename cplx_of<T>::type;

__device__ __forceinline__ float2 mk(float x, float y) { return make_float2(x, y); }
__device__ __forceinline__ double2 mk(double x, double y) { return make_double2(x, y); }

template <typename C> __device__ __forceinline__ C cadd(C a, C b) { return mk(a.x + b.x, a.y + b.y); }
template <typename C> __device__ __forceinline__ C csub(C a, C b) { return mk(a.x - b.x, a.y - b.y); }
template <typename C> __device__ __forceinline__ C cmul(C a, C b) {
  return mk(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// a * (+i)
template <typename C> __device__ __forceinline__ C cmul_i(C a) { return mk(-a.y, a.x); }
template <typename C> __device__ __forceinline__ C cconj(C a) { return mk(a.x, -a.y); }
template <typename C, typename T> __device__ __forceinline__ C cscale(C a, T s) { return mk(a.x * s, a.y * s); }

// cos / sin of 2*pi*m/32 for m < 16 (exact to double rounding).
__device__ constexpr double kCos32[16] = {
    1.0, 0.98078528040323044913, 0.92387953251128675613, 0.83146961230254523708,
    0.70710678118654752440, 0.55557023301960222474, 0.38268343236508977173, 0.19509032201612826785,
    0.0, -0.19509032201612826785, -0.38268343236508977173, -0.55557023301960222474,
    -0.70710678118654752440, -0.83146961230254523708, -0.92387953251128675613, -0.98078528040323044913};
__device__ constexpr double kSin32[16] = {
    0.0, 0.19509032201612826785, 0.38268343236508977173, 0.55557023301960222474,
    0.70710678118654752440, 0.83146961230254523708, 0.92387953251128675613, 0.98078528040323044913,
    1.0, 0.98078528040323044913, 0.92387953251128675613, 0.83146961230254523708,
    0.70710678118654752440, 0.55557023301960222474, 0.38268343236508977173, 0.19509032201612826785};

// ---------------------------------------------------------------------------
// Philox4x32-10 (Salmon et al., SC11): counter-based, stateless.
// ---------------------------------------------------------------------------
struct u32x4 { uint32_t x, y, z, w; };

__device__ __forceinline__ u32x4 philox4x32_10(u32x4 c, uint32_t k0, uint32_t k1) {
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    const uint32_t lo0 = 0xD2511F53u * c.x;
    const uint32_t hi0 = __umulhi(0xD2511F53u, c.x);
    const uint32_t lo1 = 0xCD9E8D57u * c.z;
    const uint32_t hi1 = __umulhi(0xCD9E8D57u, c.z);
    u32x4 n;
    n.x = hi1 ^ c.y ^ k0;
    n.y = lo1;
    n.z = hi0 ^ c.w ^ k1;
    n.w = lo0;
    c = n;
    k0 += 0x9E3779B9u;
    k1 += 0xBB67AE85u;
  }
  return c;
}

// The same for counters {c, 0, stream, 0} with the round keys precomputed
// (ks[r] = k0 + r 0x9E3779B9, ks[10 + r] = k1 + r 0xBB67AE85).  The mode index
// c of a padded grid fits 32 bits (at most 1025 x 2048 x 1024 draws), so what
// does not depend on it is formed once per thread: round 1 keeps one product,
// round 2 one, 18 of 20 in all.  Each 32 x 32 -> 64-bit product is one wide
// multiply (both halves); they are what a draw costs (20 measured 80 cycles a
// warp and scheduler, a quarter of the FP32 rate).
struct PhiloxLine {
  uint32_t z1, x2, z2, z3;  // key and stream parts of the first rounds' words
  uint32_t w2;
  const uint32_t* ks;
  __device__ __forceinline__ PhiloxLine(const uint32_t* ks_, uint32_t stream) : ks(ks_) {
    const uint64_t p1 = (uint64_t)0xCD9E8D57u * stream;
    const uint32_t x1 = (uint32_t)(p1 >> 32) ^ ks[0];
    const uint64_t p0 = (uint64_t)0xD2511F53u * x1;
    z1 = ks[10];
    x2 = (uint32_t)p1 ^ ks[1];
    z2 = (uint32_t)(p0 >> 32) ^ ks[11];
    w2 = (uint32_t)p0;
    z3 = w2 ^ ks[12];
  }
  __device__ __forceinline__ u32x4 operator()(uint32_t c) const {
    const uint64_t a = (uint64_t)0xD2511F53u * c;                        // round 1
    const uint64_t b = (uint64_t)0xCD9E8D57u * ((uint32_t)(a >> 32) ^ z1);  // round 2
    u32x4 v;
    v.x = (uint32_t)(b >> 32) ^ x2;
    v.y = (uint32_t)b;
    v.z = (uint32_t)a ^ z2;
    v.w = w2;
#pragma unroll
    for (int r = 2; r < 10; ++r) {
      const uint64_t p0 = (uint64_t)0xD2511F53u * v.x;
      const uint64_t p1 = (uint64_t)0xCD9E8D57u * v.z;
      u32x4 n;
      n.x = (uint32_t)(p1 >> 32) ^ v.y ^ ks[r];
      n.y = (uint32_t)p1;
      n.z = (uint32_t)(p0 >> 32) ^ (r == 2 ? z3 : v.w ^ ks[10 + r]);
      n.w = (uint32_t)p0;
      v = n;
    }
    return v;
  }
};

// Uniform in (0,1) from two 32-bit words: 52 random bits plus a half offset,
// exactly representable, never 0 or 1.
__device__ __forceinline__ double u01_d(uint32_t hi, uint32_t lo) {
  const uint64_t a = ((uint64_t)hi << 32) | lo;
  return (double)(a >> 12) * 0x1p-52 + 0x1p-53;
}
// Canonical standard normals of the padded spectrum.  Modes (kx, ky, kz) and
// (kx, ky, kz + P2/2), kz < P2/2, share one Philox draw
//   Philox(ctr = {c_lo, c_hi, stream, 0}, key),  c = kx + Hx (ky + P1 kz),
// words (x, y) feeding the first and (z, w) the second mode; each word pair
// (a, b) gives u1 = (a + 1/2) 2^-32, u2 = (b + 1/2) 2^-32 and the Box-Muller
// pair r (cos 2 pi u2, sin 2 pi u2), r = sqrt(-2 ln u1).
template <typename T> struct Normals;
template <> struct Normals<double> {
  static __device__ __forceinline__ double2 from(uint32_t a, uint32_t b) {
    const double u1 = (double)a * 0x1p-32 + 0x1p-33;
    const double u2 = (double)b * 0x1p-32 + 0x1p-33;
    const double r = sqrt(-2.0 * log(u1));
    double s, c;
    sincospi(2.0 * u2, &s, &c);
    return make_double2(r * c, r * s);
  }
};
// Hardware approximations with subnormals flushed (lg2, square root, sine and
// cosine of an argument in radians): without .ftz each carries a rescaling
// that the arguments here never need.
__device__ __forceinline__ float lg2_ftz(float x) {
  float r;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float sqrt_ftz(float x) {
  float r;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ void sincos_ftz(float x, float* s, float* c) {
  asm("sin.approx.ftz.f32 %0, %1;" : "=f"(*s) : "f"(x));
  asm("cos.approx.ftz.f32 %0, %1;" : "=f"(*c) : "f"(x));
}
template <> struct Normals<float> {
  // Single precision, hardware transcendentals: u1 is formed with one
  // rounding (relative error 2^-24, so small u1 keep their digits).  The phase
  // 2 pi (u2 - 1/2) in (-pi, pi), where the hardware sine is accurate, comes
  // from the signed word b - 2^31 by one fused multiply-add: relative error
  // 2^-24 of the reduced phase, not of u2.  The half-turn is the sign.
  static __device__ __forceinline__ float2 from(uint32_t a, uint32_t b) {
    const float u1 = __fmaf_rn((float)a, 0x1p-32f, 0x1p-33f);
    const float r = sqrt_ftz(-1.38629436111989061883f * lg2_ftz(u1));  // -2 ln 2 lg2 u1 >= 0
    const float ph = __fmaf_rn((float)(int32_t)(b ^ 0x80000000u), 6.28318530717958647692f * 0x1p-32f,
                               6.28318530717958647692f * 0x1p-33f);
    float s, c;
    sincos_ftz(ph, &s, &c);
    return make_float2(-r * c, -r * s);
  }
};

// ---------------------------------------------------------------------------
// Park-Miller (16807, 2^31-1): state after n steps from s, s in [0, 2^31-1).
// pw[b] = 16807^(2^b) mod (2^31-1).
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t pm_mulmod(uint32_t a, uint32_t b) {
  const uint64_t p = (uint64_t)a * b;
  uint64_t r = (p & 0x7FFFFFFFull) + (p >> 31);
  r = (r & 0x7FFFFFFFull) + (r >> 31);
  return (r == 0x7FFFFFFFull) ? 0u : (uint32_t)r;
}
__device__ __forceinline__ uint32_t pm_jump(uint32_t s, uint64_t n, const uint32_t* __restrict__ pw) {
  uint32_t r = s;
  int b = 0;
  while (n) {
    if (n & 1) r = pm_mulmod(r, pw[b]);
    n >>= 1;
    ++b;
  }
  return r;
}

}  // namespace scarl
