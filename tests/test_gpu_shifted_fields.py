"""Staged TPS resampling under fields that shift a volume by hundreds or
thousands of planes or rows, against the gathered path, bit for bit: shifts on
both sides of the largest that a staged walk takes, every plane still in reach
of some output voxel."""
import ctypes as C

import numpy as np
import pytest

import terawarp_b200 as tw

torch = pytest.importorskip("torch")


def _both(ctx, field, g, src, interp, want):
    hook = ctx.lib.tw_internal_set_resample_staging
    hook.restype, hook.argtypes = C.c_int, [C.c_void_p, C.c_int]
    nodes = torch.from_numpy(field).cuda()
    outs = []
    try:
        for on, launches in ((1, want), (0, 1)):
            hook(ctx.handle, on)
            dst = torch.full_like(src.to(torch.int32), 77).to(src.dtype)
            torch.cuda.synchronize()
            before = ctx.kernel_launches
            tw.warp_tps_device(ctx, nodes, g, src, dst, interp=interp)
            assert ctx.kernel_launches - before == launches
            outs.append(dst.cpu().numpy())
    finally:
        hook(ctx.handle, 1)
    np.testing.assert_array_equal(outs[0], outs[1], err_msg=f"shift {field[0, 0, 0, :3]}")
    return outs[0]


def _volume(dims, dtype, seed):
    x, y, z = dims
    return np.random.default_rng(seed).integers(0, 256 if dtype == np.uint8 else 65536, (z, y, x)).astype(dtype)


# launches of a staged job: 5, and one more where its source is first copied
# into padded rows (at least 48 Mi voxels whose rows are not multiples of 16 bytes)
@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [np.uint8, np.uint16])
@pytest.mark.parametrize("dims,g,interp,launches", [((128, 56, 2400), 16, 0, 5), ((128, 56, 2400), 4, 0, 5), ((128, 56, 2400), 64, 1, 5),
                                                    ((139, 160, 2300), 16, 0, 6)])
def test_shift_along_z(ctx, dims, g, interp, launches, dtype):
    src = torch.from_numpy(_volume(dims, dtype, g)).cuda()
    gx, gy, gz = (tw.grid_size(n, g) for n in dims)
    for dz in (400, -400, 520, -520, 600, -600, 880, -900, 1100, -1100, 1780, -1800, 2040, 2060, -2060):
        field = np.zeros((gz, gy, gx, 4), np.float32)
        field[..., :2] = 0.75, 0.5  # (no sample on a last row or column: there the two paths may round differently)
        field[..., 2] = dz + 0.25
        out = _both(ctx, field, g, src, interp, launches)
        assert out.any()  # (some samples are inside)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [np.uint8, np.uint16])
def test_shift_along_y_and_x(ctx, dtype):
    g = 16
    for dims, axis, shifts in (((128, 40000, 9), 1, (-16000, 16500, 28000, -31000, 33000, -33000, 39000)),
                               ((40000, 64, 9), 0, (-16500, 33000, -39000))):
        src = torch.from_numpy(_volume(dims, dtype, axis)).cuda()
        gx, gy, gz = (tw.grid_size(n, g) for n in dims)
        for d in shifts:
            field = np.zeros((gz, gy, gx, 4), np.float32)
            field[..., :3] = 0.25
            field[..., axis] += d
            assert _both(ctx, field, g, src, 0, 5).any()
