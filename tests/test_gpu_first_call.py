"""The first call of a context, whose tables (roots, cosines, twiddles, spectra)
are uploaded just before the kernels that read them, gives the values of a later
one, in many contexts."""
import pytest

import scarl_b200 as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("what", ["dct", "padded"])
def test_first_call_equals_the_next(what):
    import torch
    Np, P = ((16385, 3, 4), None) if what == "dct" else ((700, 9, 7), (2048, 16, 16))
    a, b = (torch.empty(Np[::-1], dtype=torch.float64, device="cuda") for _ in range(2))

    def gen(c, out):
        if what == "dct":
            S.gen_std_gauss_FFT(c, Np, tuple(float(n - 1) for n in Np), (3, 3, 3), 1, 5, 0, out=out)
        else:
            S.gen_padded(c, Np, (1, 1, 1), (30, 3, 2), 3, pad=P, seed=5, dtype=S.F64, out=out)
        c.sync()

    for i in range(40):
        with S.Context(0) as c:
            gen(c, a)
            if i == 0:
                gen(c, b)
        assert torch.equal(a, b)
