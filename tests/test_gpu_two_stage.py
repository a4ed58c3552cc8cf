"""The passes in two in-register stages.  Passes 1 and 2: every length they
serve, partial groups of kx.  Pass 3: every half length it serves, FP32 and FP64,
lines shorter and longer than its epilogue's groups of 128 and 64 values, one
and several groups of lines a warp, crop and blend, streamed moments.
Tolerances: the field gates (FP64 1e-12, FP32 1e-5 against the oracle)."""
import numpy as np
import pytest

import scarl_b200 as S

pytestmark = pytest.mark.gpu
TWO = {S.F32: 4, S.F64: 2}
HALF = [16, 24, 32, 40, 48, 56, 64, 80, 96, 112, 128, 160, 192, 224, 256, 320, 384, 448, 512, 640, 768, 896, 1024]


def rel(a, b):
    return np.linalg.norm(np.asarray(a, np.float64) - b) / np.linalg.norm(b)


@pytest.mark.parametrize("N", HALF)
@pytest.mark.parametrize("dtype,tol", [(S.F64, 1e-12), (S.F32, 1e-5)])
def test_lengths_crop(ctx, oracle, N, dtype, tol):
    if dtype == S.F64 and N > 256:
        pytest.skip("FP64 in two stages up to 256")
    ctx.tune_set(dtype, 3, N, TWO[dtype])
    try:
        for nx, ny in ((2 * N, 7), (N + 1, 16), (5, 3)):
            Np, P = (nx, ny, 5), (2 * N, 16, 8)
            ref = oracle.gen_padded(Np, P, (1, 1, 1), (6, 3, 2), 3, 0.5, 1, seed=5, stream=3)
            out = S.gen_padded(ctx, Np, (1, 1, 1), (6, 3, 2), 3, pad=P, seed=5, stream=3, dtype=dtype)
            assert rel(out, ref) < tol
    finally:
        ctx.tune_set(dtype, 3, N, -1)


@pytest.mark.parametrize("dtype,tol", [(S.F64, 1e-12), (S.F32, 1e-5)])
@pytest.mark.parametrize("xmax,pad,margi", [
    ((63, 20, 18), (64, 32, 32), 1), ((95, 20, 18), (96, 32, 32), 2), ((190, 20, 18), (128, 32, 32), 2),
    ((200, 20, 18), (192, 32, 32), 1), ((255, 20, 18), (256, 32, 32), 2), ((500, 20, 18), (448, 32, 32), 2),
    ((300, 300, 290), (224, 224, 256), 2),   # several groups of lines a warp
])
def test_blend_and_moments(ctx, oracle, dtype, tol, xmax, pad, margi):
    args = ((0, 0, 0), xmax, (4, 4, 4), (1, 1, 1), (5, 5, 5))
    topo = (2, 2, 2) if xmax[1] > 100 else (2, 1, 2)
    nb = topo[0] * topo[1] * topo[2]
    s = S.make_sample(*args, 3, margi, 1.0, 0.3, 3)
    ref, lay = oracle.generate_sample(3, *args, 3, 0.5, margi, 1.0, 0.3, 3, nb, topo, pad)
    half = pad[0] // 2
    ctx.tune_set(dtype, 3, half, TWO[dtype])
    try:
        sums = np.zeros(2)
        out, _ = S.generate_sample(ctx, s, dtype=dtype, nb_procs=nb, topo=topo, pad=pad, moments=sums)
    finally:
        ctx.tune_set(dtype, 3, half, -1)
    assert rel(out, ref) < tol
    f = out.astype(np.float64)
    # FP64 sums of n values: n 2^-53 relative at most
    assert abs(sums[0] - f.sum()) < 1e-9 * np.abs(f).sum()
    assert abs(sums[1] - (f * f).sum()) < 1e-9 * (f * f).sum()


COL = [32, 48, 64, 80, 96, 112, 128, 160, 192, 224, 256, 320, 384, 448, 512, 640, 768, 896, 1024]


@pytest.mark.parametrize("pass_", [1, 2])
@pytest.mark.parametrize("N", COL)
@pytest.mark.parametrize("dtype,tol,var", [(S.F64, 1e-12, 3), (S.F32, 1e-5, 5)])
def test_lengths_columns(ctx, oracle, N, pass_, dtype, tol, var):
    if dtype == S.F64 and N > 256:
        pytest.skip("FP64 in two stages up to 256")
    ctx.tune_set(dtype, pass_, N, var)
    try:
        for px, n in ((16, N), (32, N // 2 + 1), (64, 3)):  # Hx = 9, 17, 33: one kx past the groups
            P = (px, 8, N) if pass_ == 1 else (px, N, 8)
            Np = (px - 3, 5, n) if pass_ == 1 else (px - 3, n, 5)
            ref = oracle.gen_padded(Np, P, (1, 1, 1), (4, 3, 5), 3, 0.5, 1, seed=8, stream=2)
            out = S.gen_padded(ctx, Np, (1, 1, 1), (4, 3, 5), 3, pad=P, seed=8, stream=2, dtype=dtype)
            assert rel(out, ref) < tol
    finally:
        ctx.tune_set(dtype, pass_, N, -1)


def test_injected_normals_under_a_tuned_pass_1(ctx, oracle):
    """Injected normals run the one pass-1 variant they have, whatever the
    context is tuned to."""
    Np, P = (12, 9, 20), (16, 16, 224)
    rng = np.random.default_rng(4)
    xi = rng.standard_normal((P[2], P[1], P[0] // 2 + 1, 2))
    ctx.tune_set(S.F64, 1, 224, 3)
    try:
        out = S.gen_padded(ctx, Np, (1, 1, 1), (4, 3, 5), 3, pad=P, xi=xi, dtype=S.F64)
    finally:
        ctx.tune_set(S.F64, 1, 224, -1)
    ref = oracle.gen_padded(Np, P, (1, 1, 1), (4, 3, 5), 3, 0.5, 1, xi=xi)
    assert rel(out, ref) < 1e-12
