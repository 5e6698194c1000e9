"""Node grids of every launch form (split over warps or not, two or four nodes a
thread) agree bit for bit: the same nodes evaluated as part of a large grid and
as a small one."""
import numpy as np
import pytest

import terawarp_b200 as tw
from terawarp_b200 import synth

pytest.importorskip("torch")


@pytest.mark.gpu
@pytest.mark.parametrize("n", [4, 33, 128, 129, 257, 700])
def test_small_grids_equal_their_part_of_a_large_one(ctx, n):
    g = 8
    sub, tar = synth.lattice_landmarks((600, 500, 300), n, n)
    t = tw.tps_solve(ctx, tar, sub)
    whole = tw.tps_eval_grid(ctx, t, (83, 79, 61), g).cpu().numpy()  # 400 k nodes
    assert np.isfinite(whole).all()
    for x, y, z, i, j, k in [(1, 1, 1, 82, 0, 60), (7, 9, 5, 3, 70, 11), (33, 31, 2, 50, 0, 59), (64, 63, 27, 19, 16, 34),
                             (33, 3, 61, 0, 5, 0)]:
        part = tw.tps_eval_grid(ctx, t, (x, y, z), g, (i * g, j * g, k * g)).cpu().numpy()
        np.testing.assert_array_equal(part, whole[k:k + z, j:j + y, i:i + x])
    t.close()
