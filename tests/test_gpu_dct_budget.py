"""Literal samples under a budget: wherever tile after tile fits, the call
succeeds, also where all tiles' buffers together nearly do (the budget band
between, with host phases staged and with two long unequal axes' tables)."""
import numpy as np
import pytest

import scarl_b200 as S
from scarl_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("phases", [False, True])
def test_every_budget_above_the_smallest(ctx, oracle, phases):
    import torch
    args = ((0, 0, 0), (699, 759, 8), (4, 4, 4), (0, 0, 0.5), (5, 5, 5))
    lay = oracle.sample_layout(*args, 1, 2, (1, 1, 2))
    s = S.make_sample(*args, 1, 1, 0.5, 2.0, 3)
    n = 2 * int(np.prod(lay["Np"] // 2))
    kw = dict(generator=S.GEN_DCT, dtype=S.F64, nb_procs=2, topo=(1, 1, 2))
    if phases:
        kw["phiK"] = np.random.default_rng(4).random(n)
    ref, out = (torch.empty(tuple(lay["L"][::-1]), dtype=torch.float64, device="cuda") for _ in range(2))
    S.generate_sample(ctx, s, out=ref, **kw)
    ctx.sync()
    ran = []
    for half in range(2 * 8, 2 * 96):  # half megabytes
        with S.Context(0, budget_bytes=half << 19) as c:
            try:
                S.generate_sample(c, s, out=out, **kw)
                c.sync()
            except S.ScarlError as e:
                assert e.code == _lib.ENOMEM and not ran, half / 2
                continue
        ran.append(half)
        assert float((out - ref).norm() / ref.norm()) < 1e-13
    assert ran and ran[0] <= 2 * 40
