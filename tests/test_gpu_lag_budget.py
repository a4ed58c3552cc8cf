"""rebuild_Sk under a small budget: the blocks' partial sums give way (fewer
blocks), the values stay."""
import numpy as np
import pytest

import scarl_b200 as S
from scarl_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kb", [700, 200, 64])
def test_rebuild_sk_small_budget(ctx, kb):
    import torch
    L = (241, 201, 163)
    f = torch.rand(L[::-1], dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    ref = S.rebuild_Sk(ctx, f, L, 0.5, 0.3)
    with S.Context(0, budget_bytes=kb << 10) as c:
        out = S.rebuild_Sk(c, f, L, 0.5, 0.3)
    # sums of 512 powers and 39283 lines in another order
    assert np.abs(out - ref).max() < 1e-12 * np.abs(ref).max()


def test_rebuild_sk_budget_error():
    import torch
    f = torch.rand((163, 201, 241), dtype=torch.float64, device="cuda")
    with S.Context(0, budget_bytes=8 << 10) as c:
        with pytest.raises(S.ScarlError) as e:
            S.rebuild_Sk(c, f, (241, 201, 163), 0.5, 0.3)
    assert e.value.code == _lib.ENOMEM
