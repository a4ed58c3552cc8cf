"""Error of the literal generator's folded sums against extended precision: no
larger than that of the oracle's plain FP64 sums (its cosines are rounded once,
and half as many terms a sum leave smaller partial sums to round)."""
import numpy as np
import pytest

import scarl_b200 as S

pytestmark = pytest.mark.gpu
PI_REF = 3.1415926535898


def extended(Np, xr, cl, phi, gam):
    X = np.longdouble
    pi = 4 * np.arctan(X(1))
    s = gam.astype(X) * np.cos(2 * X(PI_REF) * phi.astype(X))
    for d in range(3):
        k = np.arange(s.shape[d]).astype(X) / X(xr[d]) / X(cl[d])
        shape = [1, 1, 1]
        shape[d] = -1
        s = s * np.sqrt(X(cl[d]) * np.exp(-X(PI_REF) * k * k)).reshape(shape)
    for d in range(3):
        i, n = np.arange(s.shape[d]), np.arange(Np[d])
        m = (i[:, None] * (2 * n[None, :] + 1)) % (4 * Np[d])
        c = 2 * np.cos(pi * m.astype(X) / (2 * Np[d]))
        c[0] = 1
        s = np.moveaxis(np.moveaxis(s, d, -1) @ c, -1, d)
    return s


@pytest.mark.parametrize("Np,cl", [((47, 38, 41), (2.0, 3.0, 2.5)), ((95, 78, 83), (0.3, 0.2, 0.25)),
                                   ((130, 65, 33), (0.05, 0.05, 0.05))])
def test_error_against_extended_precision(ctx, oracle, Np, cl):
    rng = np.random.default_rng(Np[0])
    K = [n // 2 for n in Np]
    phi = np.asfortranarray(rng.random(K))
    gam = np.asfortranarray(rng.standard_normal(K))
    xr = tuple(float(n - 1) for n in Np)
    ref = extended(Np, xr, cl, phi, gam)
    out = S.gen_std_gauss_FFT(ctx, Np, xr, cl, 1, 0, 0, phiK=phi, gammaK=gam)
    plain = oracle.gen_std_gauss_fft(Np, xr, cl, phi, gam)
    err = [float(np.sqrt(((v - ref) ** 2).sum() / (ref ** 2).sum())) for v in (out, plain)]
    print(err)
    assert err[0] <= err[1]
