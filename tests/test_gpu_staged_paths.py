"""The staged paths against the gathered one where a call would not take them by
itself, and whether calls take them at all."""
import ctypes as C

import numpy as np
import pytest

import terawarp_b200 as tw
from terawarp_b200 import synth

torch = pytest.importorskip("torch")


def _hook(ctx):
    hook = ctx.lib.tw_internal_set_resample_staging
    hook.restype, hook.argtypes = C.c_int, [C.c_void_p, C.c_int]
    return hook


MATRICES = {
    "identity": lambda d: np.eye(4),
    "half": lambda d: np.diag([2.0, 2.0, 2.0, 1.0]),
    "stretch": lambda d: np.diag([0.2, 2.5, 1.7, 1.0]),
    "flat": lambda d: np.diag([1.0, 0.0, 1.0, 1.0]),
    "affine": lambda d: synth.random_affine(3, d),
    "rotation": lambda d: synth.random_affine(4, d, rot_deg=60.0, trans=3.0),
    "quarter_reduced": lambda d: tw.make_affine(1, 0, (0, 90, 0), d) @ np.diag([1.9, 1.9, 1.9, 1.0]),
    "outside": lambda d: np.array([[1, 0, 0, 0.6 * d[0]], [0, 1, 0, -0.4 * d[1]], [0, 0, 1, 0.7 * d[2]], [0, 0, 0, 1.0]]),
}


@pytest.mark.gpu
@pytest.mark.parametrize("dims", [(64, 48, 40), (97, 61, 35), (31, 7, 3), (1, 1, 1), (288, 96, 80)])
@pytest.mark.parametrize("dtype", [np.uint8, np.uint16])
@pytest.mark.parametrize("kind", list(MATRICES))
def test_affine_boxes_that_fit_equal_gathered(ctx, dims, dtype, kind):
    x, y, z = dims
    hook = _hook(ctx)
    img = np.random.default_rng(x).integers(0, 256 if dtype == np.uint8 else 65536, (z, y, x)).astype(dtype)
    src = torch.from_numpy(img).cuda()
    M = MATRICES[kind](dims)
    for shape in ((z, y, x), (z + 5, max(1, y - 3), x + 21)):
        outs = []
        for mode in (2, 1, 0):
            hook(ctx.handle, mode)
            dst = torch.from_numpy(np.full(shape, 77, dtype)).cuda()
            torch.cuda.synchronize()
            tw.warp_affine_device(ctx, M, src, dst)
            outs.append(dst.cpu().numpy())
        hook(ctx.handle, 1)
        np.testing.assert_array_equal(outs[0], outs[2])
        np.testing.assert_array_equal(outs[1], outs[2])


# launches: 5 staged, 6 with a padded copy, 1 gathered
@pytest.mark.gpu
@pytest.mark.parametrize("dims,interp,want", [((517, 389, 253), 0, 6), ((1003, 33, 1541), 0, 6), ((517, 389, 203), 0, 1), ((1024, 512, 33), 1, 5),
                                              ((528, 485, 70), 1, 5), ((256, 256, 128), 1, 1), ((256, 256, 128), 0, 5)])
@pytest.mark.parametrize("g", [4, 16, 64])
def test_tps_calls_take_their_path(ctx, dims, interp, want, g):
    hook = _hook(ctx)
    rng = np.random.default_rng(dims[0] + g)
    src = torch.from_numpy(rng.integers(0, 256, dims[::-1]).astype(np.uint8)).cuda()
    field = rng.normal(0, 0.4, tuple(tw.grid_size(n, g) for n in dims[::-1]) + (4,)).astype(np.float32)
    field[..., :3] += (2.0, -1.0, 1.0)
    nodes = torch.from_numpy(field).cuda()
    outs = []
    for mode, launches in ((1, want), (0, 1)):
        hook(ctx.handle, mode)
        dst = torch.full_like(src, 77)
        torch.cuda.synchronize()
        before = ctx.kernel_launches
        tw.warp_tps_device(ctx, nodes, g, src, dst, interp=interp)
        assert ctx.kernel_launches - before == launches
        outs.append(dst.cpu().numpy())
    hook(ctx.handle, 1)
    np.testing.assert_array_equal(outs[0], outs[1])
