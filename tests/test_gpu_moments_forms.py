"""Streamed moments of the pass-3 kernels that an untuned context does not choose: the
FP64 engine and the FP32 register shuffles (8, 16 and 32 lanes a line where they serve
the half length 224), on the 513^3 deck, against FP64 sums of the returned field (the
same values in another order: 1e-12 relative)."""
import pytest

import scarl_b200 as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,variant", [(S.F64, 0), (S.F64, 2), (S.F32, 4), (S.F32, 5), (S.F32, 6), (S.F32, 7)])
def test_moments(ctx, dtype, variant):
    import numpy as np
    import torch
    s = S.make_sample(xMinGlob=(0, 0, 0), xMaxGlob=(512, 512, 512), corrL=(40, 20, 10), overlap=(2, 2, 2),
                      pointsPerCorrL=(41, 21, 11), corrMod=3, margiFirst=2, avg=1.0, std_dev=0.3, seedBase=0)
    out = torch.empty(513 ** 3, dtype=torch.float64 if dtype == S.F64 else torch.float32, device="cuda")
    m = np.zeros(2)
    try:
        ctx.tune_set(dtype, 3, 224, variant)
        S.generate_sample(ctx, s, dtype=dtype, nb_procs=8, topo=(2, 2, 2), pad=(448, 384, 320), out=out, moments=m)
    finally:
        ctx.tune_set(dtype, 3, 224, -1)
    f = out.double()
    ref = [float(f.sum()), float((f * f).sum())]
    assert abs(m[0] - ref[0]) <= 1e-12 * abs(ref[0]) and abs(m[1] - ref[1]) <= 1e-12 * ref[1]
