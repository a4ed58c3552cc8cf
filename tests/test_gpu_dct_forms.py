"""The literal samples' two forms on both sides of their line (a tile of 16 MB: 128^3
points), and many small tiles together beyond the L2, against the oracle.
Tolerance: FP64 sums of 64 terms along three axes, 3 x 64 x 2^-53 relative, under
the FP64 gate 1e-12.  Which form ran shows in the kernel counts."""
import numpy as np
import pytest

import scarl_b200 as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("xmax,ov,topo,batched", [
    ((127, 127, 252), (0, 0, 0.5), (1, 1, 2), True),
    ((127, 127, 254), (0, 0, 0.5), (1, 1, 2), False),
    ((205, 203, 204), (0.5, 0.5, 0.5), (3, 3, 3), True),
])
def test_forms(ctx, oracle, xmax, ov, topo, batched):
    args = ((0, 0, 0), xmax, (4, 4, 4), ov, (5, 5, 5))
    nb = topo[0] * topo[1] * topo[2]
    ref, lay = oracle.generate_sample(1, *args, 1, 0.5, 1, 0.5, 2.0, 3, nb, topo)
    assert (np.prod(lay["Np"].astype(np.int64)) <= 128 ** 3) == batched
    s = S.make_sample(*args, 1, 1, 0.5, 2.0, 3)
    ctx.profile(True)
    ctx.profile_reset()
    try:
        out, _ = S.generate_sample(ctx, s, generator=S.GEN_DCT, dtype=S.F64, nb_procs=nb, topo=topo)
        st = ctx.profile_stats()
    finally:
        ctx.profile(False)
    assert ("k_blend_gather" in st) == batched and st["k_dct_literal"][1] == (1 if batched else nb)
    assert np.linalg.norm(out - ref) < 1e-12 * np.linalg.norm(ref)
