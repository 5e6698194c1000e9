"""TPS resampling of sources that TMA cannot describe (pitches or base off 16
bytes): large ones are resampled from a copy with padded rows; against the
gathered path, bit for bit, for fields that put samples between, on and past
the last elements."""
import ctypes as C

import numpy as np
import pytest

import terawarp_b200 as tw

torch = pytest.importorskip("torch")


def _nodes(kind, gsz, g, rng):
    gx, gy, gz = gsz
    d = np.zeros((gz, gy, gx, 4), np.float32)
    if kind == "smooth":
        k, j, i = np.meshgrid(np.arange(gz), np.arange(gy), np.arange(gx), indexing="ij")
        for a in range(3):
            d[..., a] = 3.0 * np.sin(0.9 * i + a) + 2.0 * np.cos(1.1 * j - a) + 1.5 * np.sin(0.7 * k)
        d[..., :3] += rng.normal(0, 0.5, (gz, gy, gx, 3))
    elif kind == "shift":
        d[..., :3] = (2.0, -1.0, 1.0)
    elif kind == "half":  # samples at multiples of a half, some exactly on the last element
        d[..., :3] = (0.5, -0.5, 1.5)
    elif kind == "squeeze":  # q = p / 2 per axis: a linear field, reproduced by the spline
        for a, n in enumerate((gx, gy, gz)):
            shape = [1, 1, 1]
            shape[2 - a] = n
            d[..., a] = (-0.5 * (np.arange(n) - 1) * g).reshape(shape)
    elif kind == "wild":  # too wide for a staged box
        d[..., :3] = rng.normal(0, 40.0, (gz, gy, gx, 3))
    return d


@pytest.mark.gpu
@pytest.mark.parametrize("dims", [(517, 389, 253), (1003, 33, 1541)])
@pytest.mark.parametrize("dtype", [np.uint8, np.uint16])
@pytest.mark.parametrize("g", [16])
def test_padded_copy_equals_gathered(ctx, dims, dtype, g):
    x, y, z = dims
    hook = ctx.lib.tw_internal_set_resample_staging
    hook.restype, hook.argtypes = C.c_int, [C.c_void_p, C.c_int]
    rng = np.random.default_rng(x + g)
    img = rng.integers(0, 256 if dtype == np.uint8 else 65536, (z, y, x)).astype(dtype)
    buf = torch.from_numpy(np.concatenate([np.zeros(3, dtype), img.ravel()])).cuda()
    gsz = tuple(tw.grid_size(n, g) for n in dims)
    for kind in ("smooth", "half", "squeeze", "wild"):  # over 48 M voxels: the copy is taken
        nodes = torch.from_numpy(_nodes(kind, gsz, g, rng)).cuda()
        for src in (torch.from_numpy(img).cuda(), buf[3:].view(z, y, x)):  # the second: base off 16 bytes too
            outs = []
            for on in (1, 0):
                hook(ctx.handle, on)
                dst = torch.from_numpy(np.full((z, y, x), 77, dtype)).cuda()
                torch.cuda.synchronize()
                tw.warp_tps_device(ctx, nodes, g, src, dst)
                outs.append(dst.cpu().numpy())
            hook(ctx.handle, 1)
            np.testing.assert_array_equal(outs[0], outs[1], err_msg=kind)
