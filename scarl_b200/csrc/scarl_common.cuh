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
// against extended precision over 4 M random words, both ends and every
// interval's and octant's edges: ln u within 1.13e-16 of its own size (rms
// 4.7e-17), cosine and sine within 1.2e-16 (rms 2.8e-17); log has the same,
// sincospi 1.3e-16 and 3.2e-17.  A sample of four 256 x 224 x 256 grids takes 684
// us; 711 with log and sincospi, their special cases and their conversions.
//
// u = f / 2 2^k with f in [1, 2), k <= 0: k ln 2 and the logarithm of f / 2 are both
// negative, so that nothing cancels near u = 1.  Interval i of f: {c, -ln 2c}, 1 / c
// about its middle and c of 20 bits (f c - 1 is exact for the 33 bits of f), the
// last one c = 1/2; -ln 2c in two parts, the first a multiple of 2^-47 like that of
// ln 2, so that the sum k ln 2 - ln 2c of the first parts is exact.
__device__ const double2 kLogTab[64] = {
    {0x1.fc08000000000p-1, -0x1.5ee83aa241540p-1}, {0x1.f446600000000p-1, -0x1.5707a8abb8bc0p-1},
    {0x1.ecc0800000000p-1, -0x1.4f45ad35a4dc0p-1}, {0x1.e573a00000000p-1, -0x1.47a1453e8a000p-1},
    {0x1.de5d600000000p-1, -0x1.4019b2d25c700p-1}, {0x1.d77b600000000p-1, -0x1.38ae1bb197680p-1},
    {0x1.d0cb600000000p-1, -0x1.315dac0340580p-1}, {0x1.ca4b400000000p-1, -0x1.2a279850ebc40p-1},
    {0x1.c3f9000000000p-1, -0x1.230b1f8beb780p-1}, {0x1.bdd2c00000000p-1, -0x1.1c078d1ae5f00p-1},
    {0x1.b7d6c00000000p-1, -0x1.151c3aef295c0p-1}, {0x1.b203600000000p-1, -0x1.0e4893a11cc80p-1},
    {0x1.ac57000000000p-1, -0x1.078bee533c540p-1}, {0x1.a6d0200000000p-1, -0x1.00e5b51b20700p-1},
    {0x1.a16d400000000p-1, -0x1.f4aa7fe031900p-2}, {0x1.9c2d200000000p-1, -0x1.e7b447bdda780p-2},
    {0x1.970e400000000p-1, -0x1.dae72d84c8a00p-2}, {0x1.920fc00000000p-1, -0x1.ce430e8064080p-2},
    {0x1.8d30200000000p-1, -0x1.c1c61913fa100p-2}, {0x1.886e600000000p-1, -0x1.b56fa2c462900p-2},
    {0x1.83c9800000000p-1, -0x1.a93ee9c8ad600p-2}, {0x1.7f40600000000p-1, -0x1.9d32bf215ed00p-2},
    {0x1.7ad2200000000p-1, -0x1.914a84b5bf680p-2}, {0x1.767dc00000000p-1, -0x1.85853076dc000p-2},
    {0x1.7242800000000p-1, -0x1.79e25087cf780p-2}, {0x1.6e1f800000000p-1, -0x1.6e61086af1400p-2},
    {0x1.6a13c00000000p-1, -0x1.63000bb3aa180p-2}, {0x1.661ec00000000p-1, -0x1.57bf623c8cf00p-2},
    {0x1.623fa00000000p-1, -0x1.4c9df46172880p-2}, {0x1.5e75c00000000p-1, -0x1.419b4f3d5e780p-2},
    {0x1.5ac0600000000p-1, -0x1.36b692ebe0b00p-2}, {0x1.571ee00000000p-1, -0x1.2bef2c4dc8900p-2},
    {0x1.5390a00000000p-1, -0x1.21447950eaf80p-2}, {0x1.5015000000000p-1, -0x1.16b5c8bacfb80p-2},
    {0x1.4cab800000000p-1, -0x1.0c42bc7615d80p-2}, {0x1.4953a00000000p-1, -0x1.01eaeae26c680p-2},
    {0x1.460cc00000000p-1, -0x1.ef5af44dcfe00p-3}, {0x1.42d6600000000p-1, -0x1.db13cc0d48800p-3},
    {0x1.3fb0200000000p-1, -0x1.c700096eff800p-3}, {0x1.3c99600000000p-1, -0x1.b31daa75bc900p-3},
    {0x1.3991c00000000p-1, -0x1.9f6c2e7089500p-3}, {0x1.3698e00000000p-1, -0x1.8beb03b38fe00p-3},
    {0x1.33ae400000000p-1, -0x1.7898b25444700p-3}, {0x1.30d1a00000000p-1, -0x1.657556e8be700p-3},
    {0x1.2e02600000000p-1, -0x1.527e794a1b300p-3}, {0x1.2b40400000000p-1, -0x1.3fb4105991300p-3},
    {0x1.288b000000000p-1, -0x1.2d1608c868100p-3}, {0x1.25e2200000000p-1, -0x1.1aa286e23ee00p-3},
    {0x1.2345600000000p-1, -0x1.08595659e2f00p-3}, {0x1.20b4800000000p-1, -0x1.ec7470309b600p-4},
    {0x1.1e2f000000000p-1, -0x1.c886301bc0e00p-4}, {0x1.1bb4a00000000p-1, -0x1.a4e72a0b1b600p-4},
    {0x1.1945400000000p-1, -0x1.819856f40ca00p-4}, {0x1.16e0600000000p-1, -0x1.5e9526d977200p-4},
    {0x1.1486000000000p-1, -0x1.3be03a7d18c00p-4}, {0x1.1235800000000p-1, -0x1.1972e5145fa00p-4},
    {0x1.0fef000000000p-1, -0x1.eea2fc006b800p-5}, {0x1.0db2000000000p-1, -0x1.aaeded0faac00p-5},
    {0x1.0b7e600000000p-1, -0x1.67c78b2d3f400p-5}, {0x1.0954000000000p-1, -0x1.2530b2f8c8800p-5},
    {0x1.0732600000000p-1, -0x1.c63d06c14a800p-6}, {0x1.0519800000000p-1, -0x1.432ab25981000p-6},
    {0x1.0309200000000p-1, -0x1.8246da3885000p-7}, {0x1.0000000000000p-1, 0x0.0p+0}};
__device__ const double kLogTail[64] = {
    0x1.fdc69dd06becep-49, -0x1.4406284a2c39fp-50, 0x1.58a2c6521cc72p-50, -0x1.509444d8f0e83p-49,
    0x1.e4f4b0fa46764p-50, 0x1.cf7acb2d14713p-49, -0x1.ad6c61296748cp-49, 0x1.1692ce596f827p-52,
    -0x1.f814749099b49p-51, 0x1.9d4c511ce7b43p-49, -0x1.26855d451aa72p-53, -0x1.c32feb46d8ee7p-51,
    -0x1.812241434b51fp-49, 0x1.65d1a5773e100p-50, -0x1.56f2b7834ff05p-49, -0x1.5ac214be4fbf7p-51,
    -0x1.9de6e5a9bda4cp-49, -0x1.8a102e5b6643dp-49, 0x1.ddfcf88b283d2p-51, 0x1.96d6914488afap-53,
    -0x1.b6f39c7ccc1ecp-50, -0x1.d461ef2f94a4ep-49, -0x1.452b441f3e0d2p-52, -0x1.8ad99296cbc6dp-50,
    0x1.4e0cffb653f06p-51, -0x1.50b37526689c1p-49, -0x1.73b412573211bp-50, -0x1.46f6afbbf4ce1p-49,
    -0x1.f6ecfadda0cb0p-50, 0x1.5bc8b7e475979p-51, -0x1.7367b11b0cdc2p-49, 0x1.4e07764f6682ap-50,
    -0x1.efcad2851f5b3p-52, 0x1.65320905942a0p-49, -0x1.b114be4f242d6p-50, 0x1.5c46088749fbfp-49,
    -0x1.deee1199c01dfp-55, -0x1.7cd504854fc53p-49, -0x1.1e73f9bed46d4p-49, 0x1.c58c46db8fe82p-51,
    -0x1.009ac19b02d9ap-50, -0x1.ccaad56f5f767p-49, 0x1.8610ff769a574p-50, 0x1.fc342ec67c9a8p-49,
    0x1.301700f5827a4p-49, -0x1.9e2571f311bbdp-49, 0x1.8a4cdca3d82f6p-53, 0x1.b8e4a9ef7dc19p-50,
    -0x1.b10e70e60b318p-52, 0x1.891e9a1afee90p-59, -0x1.46d53dafe5901p-49, 0x1.695b9c2559e62p-50,
    0x1.5f8f872d61247p-50, -0x1.92f87e0ddb5f3p-49, -0x1.90cb9660b2485p-50, -0x1.1b388364410b8p-50,
    0x1.089f2939f3141p-50, -0x1.f82f3521ebf6cp-50, 0x1.5e328e632292ap-52, -0x1.f4fb010c6fd4fp-52,
    -0x1.14c63f750847cp-49, 0x1.dfb19b491cab3p-49, 0x1.72ef3101439fep-50, 0x0.0p+0};
template <> struct Normals<double> {
  // ln((a + 1/2) 2^-32)
  static __device__ __forceinline__ double ln_u(uint32_t a) {
    const double x = __hiloint2double(0x43300000, (int)a) - (0x1p52 - 0.5);  // a + 1/2, exact
    const int hi = __double2hiint(x), i = (hi >> 14) & 63;
    const double f = __hiloint2double((hi & 0xFFFFF) | 0x3FF00000, __double2loint(x));  // x = f 2^e
    const double2 t = __ldg(&kLogTab[i]);
    const double k = __hiloint2double(0x43300000, (hi >> 20) - 1023 - 31 + 64) - (0x1p52 + 64.0);  // e - 31, exact
    const double r = fma(f, t.x, -1.0);  // |r| <= 2^-7, exact
    double q = fma(r, -1.0 / 8.0, 1.0 / 7.0);
    q = fma(q, r, -1.0 / 6.0);
    q = fma(q, r, 1.0 / 5.0);
    q = fma(q, r, -1.0 / 4.0);
    q = fma(q, r, 1.0 / 3.0);
    q = fma(q, r, -0.5);
    const double s = fma(k, 0x1.62e42fefa3a00p-1, t.y);  // exact; 0 or larger than r
    const double w = s + r, e = r - (w - s);          // e: what w's rounding lost
    return w + fma(r * r, q, e + fma(k, -0x1.0ca86c3898d00p-49, __ldg(&kLogTail[i])));
  }
  // cos and sin of 2 pi (b + 1/2) 2^-32
  static __device__ __forceinline__ void circle(uint32_t b, double* c, double* s) {
    const uint32_t q = (b + 0x20000000u) >> 30;  // quarter turns
    const uint32_t d = b - (q << 30);            // as signed: [-2^29, 2^29)
    // the phase p + pe: 2 pi 2^-32 in two parts
    constexpr double kStep = 6.283185307179586476925 * 0x1p-32, kStepTail = 2.4492935982947064e-16 * 0x1p-32;
    const double y = __hiloint2double(0x43300000, (int)(d ^ 0x80000000u)) - (0x1p52 + 0x1p31) + 0.5;  // exact
    const double p = y * kStep, pe = fma(y, kStepTail, fma(y, kStep, -p));
    const double z = p * p;
    double u = fma(z, -1.0 / 1307674368000.0, 1.0 / 6227020800.0);
    u = fma(u, z, -1.0 / 39916800.0);
    u = fma(u, z, 1.0 / 362880.0);
    u = fma(u, z, -1.0 / 5040.0);
    u = fma(u, z, 1.0 / 120.0);
    u = fma(u, z, -1.0 / 6.0);
    const double sn = p + fma(p * z, u, pe);
    double v = fma(z, 1.0 / 20922789888000.0, -1.0 / 87178291200.0);
    v = fma(v, z, 1.0 / 479001600.0);
    v = fma(v, z, -1.0 / 3628800.0);
    v = fma(v, z, 1.0 / 40320.0);
    v = fma(v, z, -1.0 / 720.0);
    v = fma(v, z, 1.0 / 24.0);
    const double h = fma(z, -0.5, 1.0), ht = fma(z, -0.5, 1.0 - h);  // 1 - z / 2 and what its rounding lost
    const double cs = h + fma(z * z, v, fma(-p, pe, ht));
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
