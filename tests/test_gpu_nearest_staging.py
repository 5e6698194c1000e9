"""Nearest-neighbour TPS resampling from staged planes against the gathered
path, bit for bit: interior and border walks, partial units, samples on and
past the last elements."""
import ctypes as C

import numpy as np
import pytest

import terawarp_b200 as tw

torch = pytest.importorskip("torch")


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [np.uint8, np.uint16])
@pytest.mark.parametrize("g", [4, 16, 64])
@pytest.mark.parametrize("dims", [(1024, 512, 33), (528, 485, 70)])
def test_nearest_staged_equals_gathered(ctx, dims, dtype, g):
    x, y, z = dims
    hook = ctx.lib.tw_internal_set_resample_staging
    hook.restype, hook.argtypes = C.c_int, [C.c_void_p, C.c_int]
    rng = np.random.default_rng(g + x)
    src = torch.from_numpy(rng.integers(0, 256 if dtype == np.uint8 else 65536, (z, y, x)).astype(dtype)).cuda()
    gx, gy, gz = (tw.grid_size(n, g) for n in dims)
    fields = [np.full((gz, gy, gx, 4), v, np.float32) for v in (0.0, 0.5, -1.0, 2.5)]
    fields.append(rng.normal(0, 2.0, (gz, gy, gx, 4)).astype(np.float32))
    for f in fields:
        nodes = torch.from_numpy(f).cuda()
        outs = []
        for on in (1, 0):
            hook(ctx.handle, on)
            dst = torch.from_numpy(np.full((z, y, x), 77, dtype)).cuda()
            torch.cuda.synchronize()
            tw.warp_tps_device(ctx, nodes, g, src, dst, interp=1)
            outs.append(dst.cpu().numpy())
        hook(ctx.handle, 1)
        np.testing.assert_array_equal(outs[0], outs[1])
