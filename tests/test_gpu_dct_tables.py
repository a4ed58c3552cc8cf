"""The literal generator's cosine tables: kept within limits, given up where other
buffers need the room, and formed in the kernel for long axes.  Reference: the
spectrum in numpy and scipy's DCT-III.  Tolerance: FP64 sums of K terms along
three axes, 3 K 2^-53 relative."""
import numpy as np
import pytest
from scipy import fft

import scarl_b200 as S

pytestmark = pytest.mark.gpu
PI = 3.1415926535898


def reference(Np, xr, cl, phi, gam):
    sk = np.asarray(gam) * np.cos(2 * PI * np.asarray(phi))
    for d in range(3):
        k = np.arange(sk.shape[d]) / xr[d] / cl[d]
        shape = [1, 1, 1]
        shape[d] = -1
        sk = sk * np.sqrt(cl[d] * np.exp(-PI * k * k)).reshape(shape)
    full = np.zeros(Np)
    full[:sk.shape[0], :sk.shape[1], :sk.shape[2]] = sk
    return fft.dctn(full, type=3)


def check(ctx, Np, full_z=False):
    rng = np.random.default_rng(Np[0] + Np[1])
    K = [Np[0] // 2, Np[1] // 2, Np[2] if full_z else Np[2] // 2]
    phi = np.asfortranarray(rng.random(K))
    gam = np.asfortranarray(rng.standard_normal(K))
    xr, cl = tuple(float(n - 1) for n in Np), (0.02, 0.03, 0.025)
    if full_z:
        out = S.gen_std_gauss_FFT_MPI(ctx, xr, cl, L=Np, Np=Np, phiK=phi, gammaK=gam)
    else:
        out = S.gen_std_gauss_FFT(ctx, Np, xr, cl, 1, 0, 0, phiK=phi, gammaK=gam)
    ref = reference(Np, xr, cl, phi, gam)
    assert np.linalg.norm(out - ref) <= 3 * max(K) * 2.0 ** -53 * np.linalg.norm(ref)


# both sides of the largest matrix kept (8192 over half the inputs, 5793 over
# all), odd and even, few and many rows of the x step
@pytest.mark.parametrize("Np", [(8192, 3, 4), (8193, 3, 4), (8194, 17, 18), (3, 8193, 4), (4, 8303, 3), (3, 4, 8193),
                                (4, 3, 8306), (8195, 8194, 2)])
def test_cosines_formed_in_the_kernel(ctx, Np):
    check(ctx, Np)


@pytest.mark.parametrize("Np", [(3, 4, 5793), (3, 4, 5794), (4, 3, 8193)])
def test_cosines_formed_in_the_kernel_all_inputs(ctx, Np):
    check(ctx, Np, full_z=True)


def test_lognormal_long_tile(ctx, oracle):
    """The z step's lognormal output with cosines formed in the kernel; injected
    phases within 5e-8 of a quarter turn (cosine about 0) keep the exponent small:
    the two cosines there agree to 2e-16 of values of 3e-7, 1e-9 relative."""
    args = ((0, 0, 0), (6, 5, 8600), (4, 4, 4), (1, 1, 1), (5, 5, 5))
    lay = oracle.sample_layout(*args, 1, 1, (1, 1, 1))
    assert lay["Np"][2] > 8192
    n = int(np.prod(lay["Np"] // 2))
    phi = 0.25 + 1e-7 * (np.random.default_rng(2).random(n) - 0.5)
    ref, _ = oracle.generate_sample(1, *args, 1, 0.5, 2, 1.0, 0.3, 3, 1, (1, 1, 1), phiK_all=phi)
    s = S.make_sample(*args, 1, 2, 1.0, 0.3, 3)
    out, _ = S.generate_sample(ctx, s, generator=S.GEN_DCT, dtype=S.F64, phiK=phi)
    assert np.linalg.norm(np.log(out) - np.log(ref)) < 1e-8 * np.linalg.norm(np.log(ref))


def test_long_axis_small_budget():
    """40001 points: the matrix would take 3.2 GB, the roots 1.3 MB, everything
    else under 8 MB."""
    with S.Context(0, budget_bytes=10 << 20) as c:
        check(c, (40001, 3, 4))


@pytest.mark.parametrize("Np", [(131073, 2, 3), (131072, 3, 2), (140001, 4, 2)])
def test_more_inputs_than_a_grid_dimension(ctx, Np):
    check(ctx, Np)


def test_many_lengths_one_context():
    """Matrices of 40 lengths (over 20 MB together) pass through a context of 8 MB,
    and leave room for another generator's 5 MB; those of long axes (67 MB each)
    do not pile up in a large one."""
    import torch
    with S.Context(0, budget_bytes=8 << 20) as c:
        for n in range(300, 700, 10):
            check(c, (n, 5, 4))
        out = torch.empty((64, 60, 60), dtype=torch.float32, device="cuda")
        S.gen_padded(c, (60, 60, 64), (1, 1, 1), (4, 4, 4), 3, pad=(128, 128, 128), seed=1, dtype=S.F32, out=out)
        c.sync()
        check(c, (700, 5, 4))
    free0 = torch.cuda.mem_get_info()[0]
    with S.Context(0) as c:
        for n in range(5700, 5760, 5):
            check(c, (n, 2, 2))
        c.sync()
        assert free0 - torch.cuda.mem_get_info()[0] < 400 << 20
