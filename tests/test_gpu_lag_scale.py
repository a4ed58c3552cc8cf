"""rebuild_Sk at the ends of the FP64 range: the reference divides by the standard
deviation before it squares, so a field times a power of two (exact) has the same
Sk to the last bit."""
import numpy as np
import pytest

import scarl_b200 as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [-990, -600, -40, 40, 600, 1010])
def test_rebuild_sk_scaled_field(ctx, k):
    L = (40, 21, 35)
    f = np.asfortranarray(1.0 + 0.3 * np.random.default_rng(3).standard_normal(L))
    ref = S.rebuild_Sk(ctx, f, L, 1.02, 0.31)
    out = S.rebuild_Sk(ctx, np.ldexp(f, k), L, float(np.ldexp(1.02, k)), float(np.ldexp(0.31, k)))
    assert np.isfinite(ref).all() and np.abs(ref).max() > 0.1
    np.testing.assert_array_equal(out, ref)
