"""The generator's draws on chosen words: the device functions of
scarl_common.cuh compiled with the package's flags and evaluated at the edges of
their ranges and on random words."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

import scarl_b200.build as B

pytestmark = pytest.mark.gpu

SRC = r"""
#include "scarl_common.cuh"
using namespace scarl;
// per word pair: the FP32 pair, the argument of its square root
__global__ void k32(const uint32_t* a, const uint32_t* b, int n, float* o) {
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i >= n) return;
  const float2 p = Normals<float>::from(a[i], b[i]);
  o[3 * i] = p.x;
  o[3 * i + 1] = p.y;
  o[3 * i + 2] = -1.38629436111989061883f * lg2_ftz(__fmaf_rn((float)a[i], 0x1p-32f, 0x1p-33f));
}
// the split path's pair
__global__ void ksplit(const uint32_t* a, const uint32_t* b, int n, float* o) {
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i >= n) return;
  const float2 p = split_normals(a[i], b[i]);
  o[2 * i] = p.x;
  o[2 * i + 1] = p.y;
}
__global__ void kphase(const uint32_t*, const uint32_t* b, int n, float* o) {
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i < n) o[i] = split_phase(b[i]);
}
// word a as the bits of u: lg2 u and -2 ln u
__global__ void klg2(const uint32_t* a, const uint32_t*, int n, float* o) {
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i >= n) return;
  o[2 * i] = lg2_ftz(__uint_as_float(a[i]));
  o[2 * i + 1] = neg2ln(__uint_as_float(a[i]));
}
// FP64: ln((a + 1/2) 2^-32), cosine and sine of 2 pi (b + 1/2) 2^-32
__global__ void k64(const uint32_t* a, const uint32_t* b, int n, double* o) {
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i >= n) return;
  o[3 * i] = Normals<double>::ln_u(a[i]);
  Normals<double>::circle(b[i], o + 3 * i + 1, o + 3 * i + 2);
}
template <class K, class O> static int run(K k, const uint32_t* a, const uint32_t* b, int n, int w, O* out) {
  uint32_t *da, *db;
  O* d;
  if (cudaMalloc(&da, 4 * (size_t)n) || cudaMalloc(&db, 4 * (size_t)n) || cudaMalloc(&d, sizeof(O) * (size_t)n * w)) return 1;
  cudaMemcpy(da, a, 4 * (size_t)n, cudaMemcpyHostToDevice);
  cudaMemcpy(db, b, 4 * (size_t)n, cudaMemcpyHostToDevice);
  k<<<(n + 255) / 256, 256>>>(da, db, n, d);
  const int rc = cudaMemcpy(out, d, sizeof(O) * (size_t)n * w, cudaMemcpyDeviceToHost);
  cudaFree(da), cudaFree(db), cudaFree(d);
  return rc;
}
extern "C" int split(const uint32_t* a, const uint32_t* b, int n, float* o) { return run(ksplit, a, b, n, 2, o); }
extern "C" int phase(const uint32_t* a, const uint32_t* b, int n, float* o) { return run(kphase, a, b, n, 1, o); }
extern "C" int draw64(const uint32_t* a, const uint32_t* b, int n, double* o) { return run(k64, a, b, n, 3, o); }
extern "C" int lg2(const uint32_t* a, const uint32_t* b, int n, float* o) { return run(klg2, a, b, n, 2, o); }
extern "C" int draw32(const uint32_t* a, const uint32_t* b, int n, float* o) { return run(k32, a, b, n, 3, o); }
"""


@pytest.fixture(scope="module")
def dev(tmp_path_factory):
    d = tmp_path_factory.mktemp("draws")
    (d / "draws.cu").write_text(SRC)
    so = str(d / "draws.so")
    subprocess.check_call([B._nvcc()] + B.ARCH + B.COMMON + ["-shared", "-cudart", "static", str(d / "draws.cu"), "-o", so])
    return C.CDLL(so)


def call(fn, a, b, w, dt):
    a, b = np.ascontiguousarray(a, np.uint32), np.ascontiguousarray(b, np.uint32)
    out = np.empty((a.size, w), dt)
    assert fn(C.c_void_p(a.ctypes.data), C.c_void_p(b.ctypes.data), a.size, C.c_void_p(out.ctypes.data)) == 0
    return out


def words():
    """Both ends, the edges of the 64ths of every octave, the neighbourhoods of
    the multiples of an eighth turn, and random words."""
    e = [np.arange(4096), 0xFFFFFFFF - np.arange(1 << 16)]
    edges = np.array([(64 + i) << s for s in range(27) for i in range(64)], dtype=np.int64)
    e += [edges + d for d in (-1, 0, 1)]
    e += [np.arange(-2048, 2048) + (k << 29) for k in range(8)]
    e.append(np.random.default_rng(9).integers(0, 1 << 32, 1 << 20))
    return (np.concatenate(e).astype(np.int64) & 0xFFFFFFFF).astype(np.uint32)


def test_fp32_radius(dev):
    """At b = 0 the phase is -pi up to 2^-32, whose cosine rounds to -1: the first
    component is the radius sqrt(-2 ln u1).  Its root is within half a unit in the
    last place and 2^-44 relative (2^-20 units; 1e-5 with the double rounding of
    the comparison)."""
    a = words()
    o = call(dev.draw32, a, np.zeros_like(a), 3, np.float32)
    assert np.isfinite(o).all()
    r, ref = o[:, 0], np.sqrt(np.abs(o[:, 2]).astype(np.float64))
    ulp = np.spacing(np.maximum(ref, 2.0 ** -60).astype(np.float32)).astype(np.float64)
    assert (np.abs(r - ref) <= (0.5 + 1e-5) * ulp).all()


def test_log_keeps_its_sign_up_to_one(dev):
    """Every u from 1 - 2^-7 to 1, and the powers of two down to 2^-33: the
    logarithm is never positive, the argument of the radius never negative, and
    the draws at u = 1 are finite."""
    one = np.float32(1).view(np.uint32)
    bits = np.concatenate([one - np.arange(1 << 17), one - (np.arange(34) << 23)]).astype(np.uint32)
    o = call(dev.lg2, bits, bits, 2, np.float32)
    assert (o[:, 0] <= 0).all() and (o[:, 1] >= 0).all() and not np.signbit(o[:, 1]).any()
    a = np.full(4, 0xFFFFFFFF, np.uint32)
    b = np.arange(4, dtype=np.uint32) << 30
    for f, w in ((dev.draw32, 3), (dev.split, 2)):
        assert np.isfinite(call(f, a, b, w, np.float32)).all()


def test_split_phase(dev):
    """The split path's phase against 2 pi (u2 - 1/2) of the whole word: at most
    2 pi 2^-24 from the 23 bits, 2^-23 from the rounding and 2^-25 3.15 from 2 pi as
    a float (5.9e-7 in all), and no bias: the mean of 2^20 words has a standard
    error of 2.2e-10 from the truncation and less from the rounding (3e-9 allowed)."""
    b = words()
    ref = 2 * np.pi * ((b.astype(np.float64) + 0.5) * 2.0 ** -32 - 0.5)
    e = call(dev.phase, b, b, 1, np.float32)[:, 0] - ref
    assert np.abs(e).max() <= 5.9e-7
    assert abs(e[-(1 << 20):].mean()) <= 3e-9


def test_fp64_log_and_circle(dev):
    """The FP64 logarithm by table and the sine and cosine by series against
    extended precision.  Logarithm: half a unit in the last place of the result
    and 2^-5 of that for the terms added to it (at most 2^-8 of the result, three
    roundings), every table entry among the arguments.  Sine and cosine, absolute:
    half a unit below 1 (2^-54), the rounding of z / 2 (2^-55), 4.6e-17 from the
    series' first missing term and 0.6e-17 from the rest."""
    w = words()
    o = call(dev.draw64, w, w, 3, np.float64)
    one = np.longdouble(1)
    u = (w.astype(np.longdouble) + one / 2) * one / 2 ** 32
    ln = np.log(u)
    assert (np.abs(o[:, 0] - ln) <= (1 + 2.0 ** -5) * 2.0 ** -53 * np.abs(ln)).all()
    q = ((w + np.uint32(1 << 29)) >> 30).astype(np.int64)
    pi2 = 8 * np.arctan(one)
    p = ((w - (q.astype(np.uint32) << 30)).view(np.int32).astype(np.longdouble) + one / 2) / 2 ** 32 * pi2
    c, s = np.cos(p), np.sin(p)
    c, s = np.choose(q & 3, [c, -s, -c, s]), np.choose(q & 3, [s, c, -s, -c])
    tol = 2.0 ** -54 + 2.0 ** -55 + 4.6e-17 + 0.6e-17
    assert (np.abs(o[:, 1] - c) <= tol).all() and (np.abs(o[:, 2] - s) <= tol).all()
