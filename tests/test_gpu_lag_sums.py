"""rebuild_Sk at the edges of its transform lengths (N = 2n - 2 exactly, one
point below and above, odd numbers of lines, one pair of lines, the longest
line) against the oracle's windowed FFT form.  Tolerance: both sum n values per
line and transform, log2(8192) = 13 butterfly levels of 2^-53 relative each and
the window's cosine, under 1e-13 of Sk(0); the gate is the estimators' 1e-11."""
import numpy as np
import pytest

import scarl_b200 as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L", [(2, 3, 2), (9, 8, 10), (16, 17, 18), (33, 5, 34), (65, 64, 3), (129, 7, 11),
                               (130, 257, 3), (258, 3, 5), (7, 513, 514), (1025, 3, 2), (3, 1026, 5),
                               (2, 2049, 3), (2050, 2, 3), (3, 2, 4096)])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_rebuild_sk_lengths(ctx, oracle, L, dtype):
    rng = np.random.default_rng(sum(L))
    f = np.asfortranarray(1.0 + 0.3 * rng.standard_normal(L)).astype(dtype)
    for literal in (1, 0):
        ref = np.concatenate([oracle.rebuild_sk_fft(f.astype(np.float64), d, 1.02, 0.31, literal)[:L[d] // 2]
                              for d in range(3)])
        out = S.rebuild_Sk(ctx, f, L, 1.02, 0.31, tukey_literal=bool(literal))
        assert np.max(np.abs(out - ref)) < 1e-11 * np.max(np.abs(ref))
