"""The row forms of the partition of unity and of the overlap sum, bit for bit
against the oracle: one-point and whole-tile overlaps, single planes, rows
longer and shorter than a warp, three tiles a side; and uploads of small
tables that follow each other without the host waiting."""
import numpy as np
import pytest

import scarl_b200 as S

pytestmark = pytest.mark.gpu

SHAPES = [((33, 8, 7), (9, 3, 2), (3, 2, 2)), ((70, 5, 4), (1, 2, 4), (2, 2, 2)), ((12, 12, 12), (6, 6, 6), (3, 3, 3)),
          ((40, 1, 9), (8, 0, 3), (2, 1, 3)), ((1, 20, 6), (0, 5, 2), (1, 2, 2)), ((8, 8, 8), (8, 8, 8), (2, 2, 2)),
          ((65, 3, 2), (32, 1, 0), (2, 2, 1))]


@pytest.mark.parametrize("Np,No,T", SHAPES)
def test_rows_bit_exact(ctx, oracle, Np, No, T):
    rng = np.random.default_rng(7)
    nb = T[0] * T[1] * T[2]
    tiles = [np.asfortranarray(rng.standard_normal(Np)) for _ in range(nb)]
    for r in (0, nb // 2, nb - 1):
        pos = S.get_topo_pos(r, T)
        ref = oracle.apply_unity_partition(tiles[r], Np, No, pos, T)
        out = tiles[r].copy(order="F")
        S.apply_UnityPartition_mtx(ctx, out, Np, No, 1, pos, T)
        np.testing.assert_array_equal(out, ref)
    ref = np.concatenate([t.ravel(order="F") for t in oracle.add_overlap(tiles, Np, No, T)])
    out = np.concatenate([t.ravel(order="F") for t in tiles])
    S.add_overlap(ctx, out, Np, No, T)
    np.testing.assert_array_equal(out, ref)


def test_uploads_in_flight(ctx):
    """More calls in flight than staging buffers, shapes alternating, device
    outputs: each field equals the one generated alone."""
    import torch
    shapes = [(40, 33, 21), (24, 50, 30)]
    alone = []
    for i in range(24):
        Np = shapes[i % 2]
        alone.append(S.gen_std_gauss_FFT(ctx, Np, [v - 1.0 + i for v in Np], (3, 2, 4), 1, i, 0))
    outs = [torch.empty(shapes[i % 2][::-1], dtype=torch.float64, device="cuda") for i in range(24)]
    for i in range(24):
        Np = shapes[i % 2]
        S.gen_std_gauss_FFT(ctx, Np, [v - 1.0 + i for v in Np], (3, 2, 4), 1, i, 0, out=outs[i])
    ctx.sync()
    for a, o in zip(alone, outs):
        np.testing.assert_array_equal(o.cpu().numpy().ravel(), a.ravel(order="F"))
