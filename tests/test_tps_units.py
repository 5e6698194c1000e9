"""How a TPS launch is cut into work units: gathered launches have units for
every SM (no GPU); leftovers of a staged launch, few and many, equal the gathered
path bit for bit."""
import ctypes as C

import numpy as np
import pytest

import terawarp_b200 as tw
from terawarp_b200 import _lib as L

SMS = 148


def _planes(dims, g, staged):
    fn = L.load().tw_internal_tps_unit_planes
    fn.restype, fn.argtypes = C.c_int, [C.POINTER(C.c_int64), C.c_int, C.c_int, C.c_int]
    return fn((C.c_int64 * 3)(*dims), g, staged, SMS)


@pytest.mark.parametrize("g", [4, 16, 64])
@pytest.mark.parametrize("dims", [(64, 64, 64), (65, 61, 67), (129, 127, 65), (201, 197, 101), (300, 281, 97), (1025, 129, 64), (1024, 1024, 512)])
def test_gathered_launches_have_units_for_every_sm(dims, g):
    zs = _planes(dims, g, 0)
    units = lambda z: -(-dims[0] // 64) * -(-dims[1] // 16) * -(-dims[2] // z)  # noqa: E731
    assert zs == 1 or units(zs) >= 8 * SMS
    assert zs == 64 or units(2 * zs) < 8 * SMS  # and no shorter than that takes
    assert 16 <= _planes(dims, g, 1) <= 64


@pytest.mark.gpu
@pytest.mark.parametrize("wide", [0.02, 0.2, 1.0])
@pytest.mark.parametrize("dims", [(144, 48, 35), (256, 256, 128), (528, 485, 70), (1024, 1024, 128)])
def test_leftovers_equal_gathered(ctx, dims, wide):
    torch = pytest.importorskip("torch")
    g = 16
    hook = ctx.lib.tw_internal_set_resample_staging
    hook.restype, hook.argtypes = C.c_int, [C.c_void_p, C.c_int]
    rng = np.random.default_rng(dims[0])
    src = torch.from_numpy(rng.integers(0, 65536, dims[::-1]).astype(np.uint16)).cuda()
    gx, gy, gz = (tw.grid_size(n, g) for n in dims)
    field = rng.normal(0, 0.5, (gz, gy, gx, 4)).astype(np.float32)
    field[rng.random((gz, gy, gx)) < wide * 0.03] *= 90.0  # nodes whose walks are too wide to stage
    nodes = torch.from_numpy(field).cuda()
    outs = []
    for on in (1, 0):
        hook(ctx.handle, on)
        dst = torch.from_numpy(np.full(dims[::-1], 77, np.uint16)).cuda()
        torch.cuda.synchronize()
        tw.warp_tps_device(ctx, nodes, g, src, dst)
        outs.append(dst.cpu().numpy())
    hook(ctx.handle, 1)
    np.testing.assert_array_equal(outs[0], outs[1])
