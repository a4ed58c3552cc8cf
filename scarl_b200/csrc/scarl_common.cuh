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
// FP32: one packed operation for both parts (the same two roundings)
template <> __device__ __forceinline__ float2 cadd(float2 a, float2 b) { return __fadd2_rn(a, b); }
template <> __device__ __forceinline__ float2 csub(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.f, -1.f), a); }
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
// FP64: logarithm by table and series (argument reduction of P. T. P. Tang,
// "Table-driven implementation of the logarithm function in IEEE floating-point
// arithmetic", ACM TOMS 16, 1990, with 64 intervals), sine and cosine by their
// Taylor series after an exact integer reduction to an eighth turn.  Measured
// against extended precision over 4 M words and the ends of every interval: ln
// within 2.3 x 2^-53 max(1, |ln u|), the pair within 1.7e-16; the FP64 field's
// error is the same 9e-16.  With the general log and sincospi, their special
// cases and their conversions, pass 1 of four 256 x 224 x 256 grids took 365 us,
// with these 324.
//
// Interval i of [1, 2): {c, -ln c}, c the rounded inverse of its middle; the
// last one has c = 1/2 and ln 2, so that u near 1 keeps its digits.
__device__ const double2 kLogTab[64] = {
    {0x1.fc07f01fc07f0p-1, 0x1.fe02a6b106799p-8}, {0x1.f44659e4a4271p-1, 0x1.7b91b07d5b126p-6},
    {0x1.ecc07b301ecc0p-1, 0x1.39e87b9febd68p-5}, {0x1.e573ac901e574p-1, 0x1.b42dd711971b9p-5},
    {0x1.de5d6e3f8868ap-1, 0x1.16536eea37ae3p-4}, {0x1.d77b654b82c34p-1, 0x1.51b073f06183cp-4},
    {0x1.d0cb58f6ec074p-1, 0x1.8c345d6319b23p-4}, {0x1.ca4b3055ee191p-1, 0x1.c5e548f5bc743p-4},
    {0x1.c3f8f01c3f8f0p-1, 0x1.fec9131dbeabcp-4}, {0x1.bdd2b899406f7p-1, 0x1.1b72ad52f67a2p-3},
    {0x1.b7d6c3dda338bp-1, 0x1.371fc201e8f75p-3}, {0x1.b2036406c80d9p-1, 0x1.526e5e3a1b438p-3},
    {0x1.ac5701ac5701bp-1, 0x1.6d60fe719d21bp-3}, {0x1.a6d01a6d01a6dp-1, 0x1.87fa06520c911p-3},
    {0x1.a16d3f97a4b02p-1, 0x1.a23bc1fe2b561p-3}, {0x1.9c2d14ee4a102p-1, 0x1.bc286742d8cd4p-3},
    {0x1.970e4f80cb872p-1, 0x1.d5c216b4fbb94p-3}, {0x1.920fb49d0e229p-1, 0x1.ef0adcbdc5935p-3},
    {0x1.8d3018d3018d3p-1, 0x1.0402594b4d041p-2}, {0x1.886e5f0abb04ap-1, 0x1.1058bf9ae4ad4p-2},
    {0x1.83c977ab2beddp-1, 0x1.1c898c16999fbp-2}, {0x1.7f405fd017f40p-1, 0x1.2895a13de86a4p-2},
    {0x1.7ad2208e0ecc3p-1, 0x1.347dd9a987d56p-2}, {0x1.767dce434a9b1p-1, 0x1.404308686a7e4p-2},
    {0x1.724287f46debcp-1, 0x1.4be5f957778a1p-2}, {0x1.6e1f76b4337c7p-1, 0x1.5767717455a6cp-2},
    {0x1.6a13cd1537290p-1, 0x1.62c82f2b9c796p-2}, {0x1.661ec6a5122f9p-1, 0x1.6e08eaa2ba1e4p-2},
    {0x1.623fa77016240p-1, 0x1.792a55fdd47a1p-2}, {0x1.5e75bb8d015e7p-1, 0x1.842d1da1e8b18p-2},
    {0x1.5ac056b015ac0p-1, 0x1.8f11e873662c8p-2}, {0x1.571ed3c506b3ap-1, 0x1.99d958117e08ap-2},
    {0x1.5390948f40febp-1, 0x1.a484090e5bb09p-2}, {0x1.5015015015015p-1, 0x1.af1293247786bp-2},
    {0x1.4cab88725af6ep-1, 0x1.b9858969310fdp-2}, {0x1.49539e3b2d067p-1, 0x1.c3dd7a7cdad4dp-2},
    {0x1.460cbc7f5cf9ap-1, 0x1.ce1af0b85f3ecp-2}, {0x1.42d6625d51f87p-1, 0x1.d83e7258a2f3ep-2},
    {0x1.3fb013fb013fbp-1, 0x1.e24881a7c6c26p-2}, {0x1.3c995a47babe7p-1, 0x1.ec399d2468cc1p-2},
    {0x1.3991c2c187f63p-1, 0x1.f6123fa7028adp-2}, {0x1.3698df3de0748p-1, 0x1.ffd2e0857f497p-2},
    {0x1.33ae45b57bcb2p-1, 0x1.04bdf9da926d2p-1}, {0x1.30d190130d190p-1, 0x1.0986f4f573521p-1},
    {0x1.2e025c04b8097p-1, 0x1.0e44985d1cc8cp-1}, {0x1.2b404ad012b40p-1, 0x1.12f719593efbdp-1},
    {0x1.288b01288b013p-1, 0x1.179eabbd899a0p-1}, {0x1.25e22708092f1p-1, 0x1.1c3b81f713c25p-1},
    {0x1.23456789abcdfp-1, 0x1.20cdcd192ab6ep-1}, {0x1.20b470c67c0d9p-1, 0x1.2555bce98f7cap-1},
    {0x1.1e2ef3b3fb874p-1, 0x1.29d37fec2b08bp-1}, {0x1.1bb4a4046ed29p-1, 0x1.2e47436e40268p-1},
    {0x1.19453808ca29cp-1, 0x1.32b1339121d71p-1}, {0x1.16e0689427379p-1, 0x1.37117b54747b6p-1},
    {0x1.1485f0e0acd3bp-1, 0x1.3b68449fffc23p-1}, {0x1.12358e75d3033p-1, 0x1.3fb5b84d16f43p-1},
    {0x1.0fef010fef011p-1, 0x1.43f9fe2f9ce67p-1}, {0x1.0db20a88f4696p-1, 0x1.48353d1ea88dfp-1},
    {0x1.0b7e6ec259dc8p-1, 0x1.4c679afccee39p-1}, {0x1.0953f39010954p-1, 0x1.50913cc01686bp-1},
    {0x1.073260a47f7c6p-1, 0x1.54b2467999498p-1}, {0x1.05197f7d73404p-1, 0x1.58cadb5cd7989p-1},
    {0x1.03091b51f5e1ap-1, 0x1.5cdb1dc6c1765p-1}, {0x1.0000000000000p-1, 0x1.62e42fefa39efp-1}};
template <> struct Normals<double> {
  // ln((a + 1/2) 2^-32)
  static __device__ __forceinline__ double ln_u(uint32_t a) {
    const double x = __hiloint2double(0x43300000, (int)a) - (0x1p52 - 0.5);  // a + 1/2, exact
    const int hi = __double2hiint(x);
    const double f = __hiloint2double((hi & 0xFFFFF) | 0x3FF00000, __double2loint(x));  // x = f 2^e
    const double2 t = __ldg(&kLogTab[(hi >> 14) & 63]);
    const double k = __hiloint2double(0x43300000, (hi >> 20) - 1023 - 32 + 64) - (0x1p52 + 64.0);  // e - 32, exact
    const double r = fma(f, t.x, -1.0);  // |r| < 2^-7
    double q = fma(r, -1.0 / 8.0, 1.0 / 7.0);
    q = fma(q, r, -1.0 / 6.0);
    q = fma(q, r, 1.0 / 5.0);
    q = fma(q, r, -1.0 / 4.0);
    q = fma(q, r, 1.0 / 3.0);
    q = fma(q, r, -0.5);
    return fma(k, 0x1.62e42fefa39efp-1, t.y) + fma(r * r, q, r);
  }
  // cos and sin of 2 pi (b + 1/2) 2^-32
  static __device__ __forceinline__ void circle(uint32_t b, double* c, double* s) {
    const uint32_t q = (b + 0x20000000u) >> 30;  // quarter turns
    const uint32_t d = b - (q << 30);            // as signed: [-2^29, 2^29)
    constexpr double kStep = 6.283185307179586476925 * 0x1p-32;
    const double p = fma(__hiloint2double(0x43300000, (int)(d ^ 0x80000000u)) - (0x1p52 + 0x1p31), kStep, 0.5 * kStep);
    const double z = p * p;
    double u = fma(z, -1.0 / 1307674368000.0, 1.0 / 6227020800.0);
    u = fma(u, z, -1.0 / 39916800.0);
    u = fma(u, z, 1.0 / 362880.0);
    u = fma(u, z, -1.0 / 5040.0);
    u = fma(u, z, 1.0 / 120.0);
    u = fma(u, z, -1.0 / 6.0);
    const double sn = fma(p * z, u, p);
    double v = fma(z, 1.0 / 20922789888000.0, -1.0 / 87178291200.0);
    v = fma(v, z, 1.0 / 479001600.0);
    v = fma(v, z, -1.0 / 3628800.0);
    v = fma(v, z, 1.0 / 40320.0);
    v = fma(v, z, -1.0 / 720.0);
    v = fma(v, z, 1.0 / 24.0);
    v = fma(v, z, -0.5);
    const double cs = fma(v, z, 1.0);
    const double cq = (q & 1) ? sn : cs, sq = (q & 1) ? cs : sn;  // q = 1: (-s, c), 2: (-c, -s), 3: (s, -c)
    *c = __hiloint2double(__double2hiint(cq) ^ (int)(((q + 1) & 2) << 30), __double2loint(cq));
    *s = __hiloint2double(__double2hiint(sq) ^ (int)((q & 2) << 30), __double2loint(sq));
  }
  static __device__ __forceinline__ double2 from(uint32_t a, uint32_t b) {
    const double r = sqrt(-2.0 * ln_u(a));
    double s, c;
    circle(b, &c, &s);
    return make_double2(r * c, r * s);
  }
};

// Hardware approximations with subnormals flushed (lg2, sine and cosine of an
// argument in radians; the split path's square root): without .ftz each carries
// a rescaling that the arguments here never need.
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
// sqrt(x) of x = 0 or normal by one Newton step (Heron's) on x times the
// hardware reciprocal root, with the residual x - r^2 exact: within half a unit
// in the last place and 2^-44, where the bare hardware root is off by up to 2^-23.
// 1.52 ms a sample of two by two tiles padded to 512^3; 1.48 with the bare root,
// 1.58 with sqrtf and its branch to a slow path.
__device__ __forceinline__ float sqrt_newton(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(fmaxf(x, 0x1p-100f)));
  const float r = x * y;
  return __fmaf_rn(__fmaf_rn(-r, r, x), 0.5f * y, r);
}
__device__ __forceinline__ void sincos_ftz(float x, float* s, float* c) {
  asm("sin.approx.ftz.f32 %0, %1;" : "=f"(*s) : "f"(x));
  asm("cos.approx.ftz.f32 %0, %1;" : "=f"(*c) : "f"(x));
}
// -2 ln u for 0 < u <= 1.  The hardware logarithm's error is absolute, 2^-22 for
// u above 1/2, so its sign near u = 1 is not the specification's to promise: the
// magnitude is taken (it costs nothing), and no root sees a negative.
__device__ __forceinline__ float neg2ln(float u) { return fabsf(-1.38629436111989061883f * lg2_ftz(u)); }
template <> struct Normals<float> {
  // Single precision, hardware logarithm, sine and cosine: u1 is formed with
  // one rounding (relative error 2^-24, so small u1 keep their digits).  The phase
  // 2 pi (u2 - 1/2) in (-pi, pi), where the hardware sine is accurate, comes
  // from the signed word b - 2^31 by one fused multiply-add: relative error
  // 2^-24 of the reduced phase, not of u2.  The half-turn is the sign.
  static __device__ __forceinline__ float2 from(uint32_t a, uint32_t b) {
    const float u1 = __fmaf_rn((float)a, 0x1p-32f, 0x1p-33f);
    const float r = sqrt_newton(neg2ln(u1));
    const float ph = __fmaf_rn((float)(int32_t)(b ^ 0x80000000u), 6.28318530717958647692f * 0x1p-32f,
                               6.28318530717958647692f * 0x1p-33f);
    float s, c;
    sincos_ftz(ph, &s, &c);
    return make_float2(-r * c, -r * s);
  }
};

// The canonical Box-Muller pair of Normals<float> (u1 = (a + 1/2) 2^-32,
// u2 = (b + 1/2) 2^-32, r (cos 2 pi u2, sin 2 pi u2), r = sqrt(-2 ln u1)) at
// the split path's accuracy: the phase 2 pi (u2 - 1/2) from the top 23 bits of
// b as the mantissa of m in [1, 2), without a conversion; m - 3/2 is exact, the
// half step comes in with the product.  Phase error up to 5.8e-7 (the 23 bits
// 3.7e-7, the rounding 1.2e-7, 2 pi as a float 0.9e-7) and 0 on average, far below
// the 2^-17 of the BF16 split.
__device__ __forceinline__ float split_phase(uint32_t b) {
  constexpr float k2Pi = 6.28318530717958647692f;
  return __fmaf_rn(__uint_as_float(0x3F800000u | (b >> 9)) - 1.5f, k2Pi, 0x1p-24f * k2Pi);
}
__device__ __forceinline__ float2 split_normals(uint32_t a, uint32_t b) {
  const float u1 = __fmaf_rn((float)a, 0x1p-32f, 0x1p-33f);
  const float r = sqrt_ftz(neg2ln(u1));
  float s, c;
  sincos_ftz(split_phase(b), &s, &c);
  return make_float2(-r * c, -r * s);
}

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
