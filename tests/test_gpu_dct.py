"""The literal DCT generator's matrix products at the edges of their tiles, and
both forms of its blend (one gather over tiles held together; each tile's
output stage) against the oracle.  Tolerance: FP64 sums of at most 200 terms
along three axes, 3 x 200 x 2^-53 = 7e-14 relative, under the FP64 gate 1e-12."""
import numpy as np
import pytest

import scarl_b200 as S

pytestmark = pytest.mark.gpu
TOL64 = 1e-12


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


# rows of 16 / 32 / 64 (folded lengths 16, 32, 64 are N = 31..33, 63..65,
# 127..129), columns of 64, inputs of 16, odd and even lengths, one input
@pytest.mark.parametrize("Np", [(2, 2, 2), (3, 2, 5), (2, 64, 3), (65, 3, 33), (31, 32, 33), (63, 64, 65),
                                (127, 7, 129), (128, 126, 5), (130, 34, 66), (9, 297, 17), (64, 65, 200)])
def test_dct_tile_edges(ctx, oracle, Np):
    rng = np.random.default_rng(5)
    K = [n // 2 for n in Np]
    phi = np.asfortranarray(rng.random(K))
    gam = np.asfortranarray(rng.standard_normal(K))
    xr = tuple(float(n - 1) for n in Np)
    ref = oracle.gen_std_gauss_fft(Np, xr, (3, 2, 4), phi, gam)
    out = S.gen_std_gauss_FFT(ctx, Np, xr, (3, 2, 4), 1, 0, 0, phiK=phi, gammaK=gam)
    assert rel(out, ref) < TOL64


# below 64 MB of tiles together the gather; above it tile after tile
@pytest.mark.parametrize("xmax,ov,topo,margi", [
    ((30, 25, 41), (1, 1, 1), (2, 1, 3), 1),
    ((33, 21, 18), (0, 0, 0), (3, 2, 1), 1),        # neighbours share one plane
    ((20, 20, 20), (2, 1, 1.5), (2, 2, 2), 1),
    ((214, 203, 199), (1, 1, 2), (1, 2, 2), 1),
    ((211, 205, 201), (0, 1, 0), (2, 1, 2), 1),
])
def test_dct_blend_forms(ctx, oracle, xmax, ov, topo, margi):
    args = ((0, 0, 0), xmax, (4, 4, 4), ov, (5, 5, 5))
    nb = topo[0] * topo[1] * topo[2]
    ref, lay = oracle.generate_sample(1, *args, 1, 0.5, margi, 0.5, 2.0, 3, nb, topo)
    s = S.make_sample(*args, 1, margi, 0.5, 2.0, 3)
    out, glay = S.generate_sample(ctx, s, generator=S.GEN_DCT, dtype=S.F64, nb_procs=nb, topo=topo)
    np.testing.assert_array_equal(glay["L"], lay["L"])
    assert rel(out, ref) < TOL64


def test_dct_lognormal_tile_after_tile(ctx, oracle):
    """The output stage with the lognormal marginal; injected phases of 1/4
    (cosine about 0) keep the exponent small."""
    args = ((0, 0, 0), (206, 204, 202), (4, 4, 4), (1, 1, 1), (5, 5, 5))
    lay = oracle.sample_layout(*args, 1, 2, (1, 1, 2))
    n = int(np.prod(lay["Np"] // 2)) * 2
    phi = 0.25 + 1e-5 * (np.random.default_rng(2).random(n) - 0.5)
    ref, _ = oracle.generate_sample(1, *args, 1, 0.5, 2, 1.0, 0.5, 3, 2, (1, 1, 2), phiK_all=phi)
    s = S.make_sample(*args, 1, 2, 1.0, 0.5, 3)
    out, _ = S.generate_sample(ctx, s, generator=S.GEN_DCT, dtype=S.F64, nb_procs=2, topo=(1, 1, 2), phiK=phi)
    # cos of phases near a quarter turn: the two math libraries' cosines agree
    # to an ulp of 1, 2e-16 of values of 3e-5: 1e-11 relative
    assert rel(out - 1.0, ref - 1.0) < 1e-9


def test_dct_small_budget(oracle):
    """A context whose budget holds one tile's buffers but not all tiles'
    together generates tile after tile."""
    args = ((0, 0, 0), (90, 90, 90), (4, 4, 4), (1, 1, 1), (5, 5, 5))
    ref, _ = oracle.generate_sample(1, *args, 1, 0.5, 1, 0.5, 2.0, 3, 8, (2, 2, 2))
    s = S.make_sample(*args, 1, 1, 0.5, 2.0, 3)
    # field 91^3: 6 MB staged; a 48^3 tile's spectrum and steps under 2 MB, 8
    # tiles' buffers together over 12 MB
    with S.Context(0, budget_bytes=12 << 20) as c:
        out, _ = S.generate_sample(c, s, generator=S.GEN_DCT, dtype=S.F64, nb_procs=8, topo=(2, 2, 2))
    assert rel(out, ref) < TOL64
