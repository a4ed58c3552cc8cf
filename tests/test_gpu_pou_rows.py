"""Partition of unity on fields of about 2^31 rows (a row index and the walk's last
step beyond 32 bits): 17 GB of one point a row, against the product of the axes'
factors.  Tolerance: two square roots and their product against one root, 4 x 2^-53."""
import pytest

import scarl_b200 as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ny,nz", [(32767, 65536), (65536, 32769)])
def test_two_to_the_31_rows(ctx, ny, nz):
    import torch
    if torch.cuda.mem_get_info()[0] < 40 << 30:
        pytest.skip("needs 40 GB of free device memory")

    def factors(Np, No, pos, shape):
        f = torch.ones(Np[::-1], dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        S.apply_UnityPartition_mtx(ctx, f, Np, No, 1, pos, shape)
        ctx.sync()
        return f

    wy = factors((1, ny, 1), (0, 5, 0), (0, 1, 0), (1, 3, 1)).flatten()
    wz = factors((1, 1, nz), (0, 0, 7), (0, 0, 1), (1, 1, 2)).flatten()
    out = factors((1, ny, nz), (0, 5, 7), (0, 1, 1), (1, 3, 2)).reshape(nz, ny)
    for z in range(0, nz, 4096):
        ref = wz[z:z + 4096, None] * wy[None, :]
        assert bool(((out[z:z + 4096] - ref).abs() <= 4 * 2.0 ** -53 * ref).all())
    del out
    torch.cuda.empty_cache()
