"""The affine landmark fit at the sizes where its partition of the landmarks
changes: part of a warp, whole warps, one landmark past the CTA's 256, several
per thread."""
import numpy as np
import pytest

import terawarp_b200 as tw
from oracle import oracle as O
from terawarp_b200 import synth


@pytest.mark.gpu
@pytest.mark.parametrize("n", [6, 31, 32, 33, 255, 256, 257, 769, 4096])
def test_affine_fit_sizes(ctx, n):
    # the fit's eigenvector carries at most ~13 eps |A| / gap ~ 1e-13 of
    # relative error in either implementation (|A| / gap of the normalised
    # normal matrix is below 40 for these points), on coordinates below 1e3:
    # 1e-10; 1e-8 leaves room for a badly placed sample at n = 6
    M = synth.random_affine(n, (700, 600, 300))
    sub, tar = synth.affine_landmarks(M, (700, 600, 300), n, n + 1)
    np.testing.assert_allclose(tw.fit_affine(ctx, tar, sub), O.affine_fit(tar, sub), rtol=0, atol=1e-8)
