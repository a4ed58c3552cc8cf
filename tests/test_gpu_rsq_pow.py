"""Powers b^(-n/2) of the Matern amplitudes (gen_kernels.cuh), compiled with the
package's flags, against extended precision: within half a unit in the last
place, 2^-14 of one for the terms left out, and 2^-10 for the reference's own
rounding against FP64."""
import ctypes as C
import subprocess

import numpy as np
import pytest

import scarl_b200.build as B

pytestmark = pytest.mark.gpu

SRC = r"""
#include "gen_kernels.cuh"
using namespace scarl;
template <typename T> __global__ void kp(const T* b, int n, int m, T* o) {
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i < n) o[i] = rsq_pow<T>(b[i], m);
}
template <typename T> static int run(const T* b, int n, int m, T* o) {
  T *d, *r;
  if (cudaMalloc(&d, sizeof(T) * (size_t)n) || cudaMalloc(&r, sizeof(T) * (size_t)n)) return 1;
  cudaMemcpy(d, b, sizeof(T) * (size_t)n, cudaMemcpyHostToDevice);
  kp<T><<<(n + 255) / 256, 256>>>(d, n, m, r);
  const int rc = cudaMemcpy(o, r, sizeof(T) * (size_t)n, cudaMemcpyDeviceToHost);
  cudaFree(d), cudaFree(r);
  return rc;
}
extern "C" int pow32(const float* b, int n, int m, float* o) { return run(b, n, m, o); }
extern "C" int pow64(const double* b, int n, int m, double* o) { return run(b, n, m, o); }
"""


@pytest.fixture(scope="module")
def dev(tmp_path_factory):
    d = tmp_path_factory.mktemp("rsq")
    (d / "rsq.cu").write_text(SRC)
    so = str(d / "rsq.so")
    subprocess.check_call([B._nvcc()] + B.ARCH + B.COMMON + ["-shared", "-cudart", "static", str(d / "rsq.cu"), "-o", so])
    return C.CDLL(so)


@pytest.mark.parametrize("n", range(2, 9))
@pytest.mark.parametrize("dt", [np.float32, np.float64])
def test_rsq_pow(dev, dt, n):
    rng = np.random.default_rng(n)
    b = np.concatenate([[1.0], 1 + np.arange(1, 200) * np.finfo(dt).eps, 4.0 ** np.arange(11),
                        2.0 ** rng.uniform(0, 22, 1 << 16)]).astype(dt)  # 22: (pi 40)^2 and three axes, times 85
    o = np.empty_like(b)
    f = dev.pow32 if dt == np.float32 else dev.pow64
    assert f(C.c_void_p(b.ctypes.data), b.size, n, C.c_void_p(o.ctypes.data)) == 0
    ref = b.astype(np.longdouble) ** (np.longdouble(-n) / 2)
    ulp = np.spacing(ref.astype(dt)).astype(np.longdouble)
    assert (np.abs(o - ref) <= (0.5 + 2.0 ** -14 + 2.0 ** -10) * ulp).all()
