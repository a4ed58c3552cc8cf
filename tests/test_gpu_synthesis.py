"""The spectrum synthesis of pass 1 against the oracle: powers of 1/sqrt (half-
integer Matern orders) at both ends of their range and general powers beside
them, the Philox counters at the ends of key and stream, every way a thread's
draws fall on its first stage.  Tolerances: the FP64 and FP32 field gates."""
import numpy as np
import pytest

import scarl_b200 as S

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.linalg.norm(np.asarray(a, np.float64) - b) / np.linalg.norm(b)


@pytest.mark.parametrize("nu", [0.49, 1.0, 1.5, 2.5, 4.5, 6.5, 7.5])
@pytest.mark.parametrize("P", [(32, 16, 64), (32, 16, 320)])
def test_matern_orders(ctx, oracle, nu, P):
    Np, cl = (20, 11, P[2] // 2 + 3), (9.0, 4.0, 6.0)
    ref = oracle.gen_padded(Np, P, (1, 1, 1), cl, 2, nu, 1, seed=5, stream=1)
    for dtype, tol in ((S.F64, 1e-12), (S.F32, 1e-5), (S.F32 | S.SPLIT_BF16, 1e-5)):
        out = S.gen_padded(ctx, Np, (1, 1, 1), cl, 2, nu, pad=P, seed=5, stream=1, dtype=dtype)
        assert rel(out, ref) < tol


@pytest.mark.parametrize("seed,stream", [(0, 0), (2 ** 64 - 1, 2 ** 32 - 1), (2 ** 32, 1), (1, 2 ** 31)])
@pytest.mark.parametrize("n2", [8, 16, 32, 48, 128, 224, 256, 2048])
def test_counters(ctx, oracle, seed, stream, n2):
    P = (16, 8, n2)
    Np = (7, 5, n2 - 3)
    ref = oracle.gen_padded(Np, P, (1, 1, 1), (3, 3, 5), 3, 0.5, 1, seed=seed, stream=stream)
    for dtype, tol in ((S.F64, 1e-12), (S.F32, 1e-5), (S.F32 | S.SPLIT_BF16, 1e-5)):
        out = S.gen_padded(ctx, Np, (1, 1, 1), (3, 3, 5), 3, pad=P, seed=seed, stream=stream, dtype=dtype)
        assert rel(out, ref) < tol
