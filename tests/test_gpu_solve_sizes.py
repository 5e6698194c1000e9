"""The landmark solve at the sizes where its tiling changes: one tile, its last
row, one row into the next tile, the first sizes with look-ahead rows, tiles
for more than one block of the grid."""
import numpy as np
import pytest

import terawarp_b200 as tw
from oracle import oracle as O
from terawarp_b200 import synth


@pytest.mark.gpu
@pytest.mark.parametrize("n", [5, 67, 68, 69, 131, 132, 133, 197, 261, 325, 389, 453, 1345])
def test_solve_sizes(ctx, n):
    # both solve the same system by backward-stable factorisations in FP64:
    # coefficients agree to about eps times the condition number (below 1e5
    # here: |K| up to n * 700, smallest eigenvalue at least lambda = 0.2), taken
    # relative to the largest coefficient
    sub, tar = synth.lattice_landmarks((700, 600, 300), n, n)
    t = tw.tps_solve(ctx, tar, sub)
    c, d = t.coeffs()
    t.close()
    rc, rd = O.tps_solve(tar, sub)
    tol = 2.2e-16 * (700.0 * n / 0.2)
    np.testing.assert_allclose(c, rc, rtol=0, atol=tol * np.abs(rc).max())
    np.testing.assert_allclose(d, rd, rtol=0, atol=tol * np.abs(rd).max())


@pytest.mark.gpu
def test_solve_repeats_bit_for_bit(ctx):
    # tiles are claimed in whatever order the CTAs come; the result does not depend on it
    sub, tar = synth.lattice_landmarks((700, 600, 300), 900, 3)
    first = None
    for _ in range(5):
        t = tw.tps_solve(ctx, tar, sub)
        c, d = t.coeffs()
        t.close()
        if first is None:
            first = (c, d)
        np.testing.assert_array_equal(c, first[0])
        np.testing.assert_array_equal(d, first[1])
