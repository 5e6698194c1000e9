"""Node grids a few nodes deep: how they are dealt to threads (no GPU), and that
they agree bit for bit with the same nodes of a deep grid."""
import ctypes as C

import numpy as np
import pytest

import terawarp_b200 as tw
from terawarp_b200 import _lib as L
from terawarp_b200 import synth


def _form(gsz, n, sms=148):
    fn = L.load().tw_internal_eval_form
    fn.restype, fn.argtypes = None, [C.POINTER(C.c_int64), C.c_int, C.c_int, C.POINTER(C.c_int)]
    out = (C.c_int * 3)()
    fn((C.c_int64 * 3)(*gsz), n, sms, out)
    return tuple(out)


@pytest.mark.parametrize("n", [16, 2000])
@pytest.mark.parametrize("gx,gy", [(515, 515), (259, 259), (131, 131), (67, 700), (1001, 13)])
@pytest.mark.parametrize("gz", [1, 2, 3, 4, 5, 6, 7, 9, 13, 35, 131])
def test_few_nodes_are_evaluated_in_vain(gx, gy, gz, n):
    npt, split, axis = _form((gx, gy, gz), n)
    run = (gx, gy, gz)[axis]
    assert npt in (2, 4) and split in (1, 8) and axis in (0, 2)
    assert -(-run // npt) * npt <= 1.15 * run


def test_deep_grids_run_along_z():
    for gsz in [(131, 131, 67), (83, 79, 61), (67, 67, 35), (1, 1, 61), (3, 900, 48)]:
        assert _form(gsz, 500)[2] == 2


@pytest.mark.gpu
@pytest.mark.parametrize("n", [4, 129, 700])
def test_flat_grids_equal_their_part_of_a_deep_one(ctx, n):
    g = 8
    sub, tar = synth.lattice_landmarks((2000, 1800, 300), n, n)
    t = tw.tps_solve(ctx, tar, sub)
    whole = tw.tps_eval_grid(ctx, t, (259, 243, 40), g).cpu().numpy()
    assert _form((259, 243, 40), n)[2] == 2
    forms = set()
    # thread forms of all three sizes along x, runs that end at, before and after the row's end
    for x, y, z, i, j, k in [(259, 243, 5, 0, 0, 7), (258, 240, 9, 1, 2, 31), (257, 243, 1, 0, 0, 39), (260 - 4, 241, 6, 3, 1, 0), (101, 99, 5, 50, 9, 3),
                             (131, 31, 3, 7, 9, 20), (67, 9, 1, 0, 3, 39)]:
        form = _form((x, y, z), n)
        assert form[2] == 0
        forms.add(form)
        part = tw.tps_eval_grid(ctx, t, (x, y, z), g, (i * g, j * g, k * g)).cpu().numpy()
        np.testing.assert_array_equal(part, whole[k:k + z, j:j + y, i:i + x])
    assert len(forms) >= 2 + (n > 128)
    t.close()
