"""Pass 3's bounded wait for its line copies has one outcome for a warp: with the
test hook the odd lanes count every copy as late although it has landed, and
every lane has to leave (nothing written, SCARL_ETIMEOUT reported) and the
context to generate correctly afterwards.  Every kernel that waits so: the
two-stage form with and without aliased areas, FP32 and FP64, several groups of
lines a warp, and the register-shuffle form."""
import pytest

import scarl_b200 as S
from scarl_b200 import _lib

pytestmark = pytest.mark.gpu
TWO = {S.F32: 4, S.F64: 2}       # the two-stage variant of pass 3
SHFL16 = 6                       # register shuffles, 16 lanes a line


@pytest.mark.parametrize("dt,N,v,lines", [
    (S.F32, 256, TWO[S.F32], (6, 5)), (S.F32, 384, TWO[S.F32], (6, 5)), (S.F64, 112, TWO[S.F64], (7, 3)),
    (S.F64, 224, TWO[S.F64], (7, 3)), (S.F32, 64, TWO[S.F32], (300, 700)), (S.F32, 256, SHFL16, (6, 5)),
])
def test_late_copies_leave_every_lane(ctx, dt, N, v, lines):
    import torch
    td = torch.float32 if dt == S.F32 else torch.float64
    Np = (N + 5, lines[0], lines[1])
    P = (2 * N, 512 if lines[0] > 8 else 8, 1024 if lines[1] > 8 else 8)
    kw = dict(pad=P, seed=5, stream=3, dtype=dt)
    out = torch.full(Np[::-1], -7.0, dtype=td, device="cuda")
    torch.cuda.synchronize()
    try:
        ctx.tune_set(dt, 3, N, v)
        ctx.tc_wait_test(True)
        with pytest.raises(S.ScarlError) as e:
            S.gen_padded(ctx, Np, (1, 1, 1), (6, 3, 2), 3, out=out, **kw)
            ctx.sync()
        assert e.value.code == _lib.ETIMEOUT
        assert bool((out == -7.0).all())
        ctx.tc_wait_test(False)
        S.gen_padded(ctx, Np, (1, 1, 1), (6, 3, 2), 3, out=out, **kw)
        ctx.tune_set(dt, 3, N, 0)  # the shared-memory engine
        ref = torch.empty_like(out)
        S.gen_padded(ctx, Np, (1, 1, 1), (6, 3, 2), 3, out=ref, **kw)
        ctx.sync()
        assert float((out - ref).norm() / ref.norm()) < (1e-6 if dt == S.F32 else 1e-14)
    finally:
        ctx.tc_wait_test(False)
        ctx.tune_set(dt, 3, N, -1)
