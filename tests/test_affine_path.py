"""Which affine warps are sampled from staged boxes and which gather (no GPU):
the cases lie well away from where the two take the same time."""
import ctypes as C

import numpy as np
import pytest

import terawarp_b200 as tw
from terawarp_b200 import _lib as L

GATHERED, TMA, GRANULES = 0, 1, 2
ALIGNED, RAGGED = (1024, 1024, 512), (1021, 1019, 509)


def _path(A, dtype, dims, out=None):
    fn = L.load().tw_internal_affine_path
    fn.restype, fn.argtypes = C.c_int, [C.POINTER(C.c_double), C.c_int, C.POINTER(C.c_int64), C.POINTER(C.c_int64)]
    M = np.eye(4)
    M[:3, :3] = A
    M[:3, 3] = 0.5 * (np.array(dims) - 1) - A @ (0.5 * (np.array(out or dims) - 1))  # centre onto centre
    return fn((C.c_double * 16)(*M.ravel()), dtype, (C.c_int64 * 3)(*dims), (C.c_int64 * 3)(*(out or dims)))


def _rot(angles, s=1.0):
    return tw.make_affine(1, 0, angles, ALIGNED)[:3, :3] * s


def _reduced(dims, by):
    return tuple(int(n / b) for n, b in zip(dims, by))


@pytest.mark.parametrize("dtype", [1, 2])
@pytest.mark.parametrize("A", [np.eye(3), np.eye(3) * 1.25, np.diag([1, 1, 2]), _rot((15, 15, 15)), _rot((0, 0, 45), 1.4), _rot((0, 90, 0)),
                               _rot((45, 45, 45)), _rot((15, 15, 15), 1.4)])
def test_aligned_sources_are_staged(A, dtype):
    assert _path(A, dtype, ALIGNED) == TMA


@pytest.mark.parametrize("dtype", [1, 2])
@pytest.mark.parametrize("A", [np.eye(3) * 0.5, _rot((15, 15, 15)), _rot((0, 0, 45)), _rot((0, 90, 0)), _rot((45, 45, 45)), _rot((90, 0, 0))])
def test_ragged_sources_are_staged_by_granules(A, dtype):
    assert _path(A, dtype, RAGGED) == GRANULES


@pytest.mark.parametrize("dtype", [1, 2])
@pytest.mark.parametrize("A,by", [(np.eye(3) * 1.75, (1.75, 1.75, 1.75)), (np.eye(3) * 2.0, (2, 2, 2)), (np.diag([1, 1, 4]), (1, 1, 4)),
                                  (np.diag([1, 2, 2]), (1, 2, 2)), (_rot((10, 0, 0), 1.8), (1.8, 1.8, 1.8)), (_rot((1, 1, 1), 2.0), (2, 2, 2))])
def test_reductions_of_ragged_sources_gather(A, by, dtype):
    # 1.5 to 2.5 times the time when staged
    assert _path(A, dtype, RAGGED, _reduced(RAGGED, by)) == GATHERED


def test_reductions_of_aligned_sources():
    for s, dtype, want in ((2.25, 1, GATHERED), (1.75, 2, TMA), (1.5, 1, TMA)):  # us: 246 and 303 staged, 678 and 582, 601 and 515
        assert _path(np.eye(3) * s, dtype, ALIGNED, _reduced(ALIGNED, (s, s, s))) == want


def test_outputs_mostly_outside_the_source():
    # a quarter turn about y with a reduction by 2: seven eighths of an output as
    # large as the source lie outside it, where gathering costs little
    dims = (512, 512, 256)
    assert _path(_rot((0, 90, 0), 2.0), 2, dims) == GATHERED
    assert _path(_rot((0, 90, 0), 2.0), 2, dims, _reduced(dims, (4, 2, 1))) == TMA


def test_extreme_matrices_gather():
    for A in (np.eye(3) * 20.0, np.full((3, 3), np.nan), np.eye(3) * 1e30, np.eye(3) + 1e300):
        assert _path(A, 1, ALIGNED) == GATHERED
