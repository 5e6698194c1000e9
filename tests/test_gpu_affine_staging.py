"""Affine tiles staged in shared memory against the gathered path, bit for
bit: rows whose pitch is and is not a multiple of 16 bytes, volumes smaller
than a tile, partial tiles, resized outputs, one and two stages, sources that
TMA boxes, copies by granules or neither can take."""
import ctypes as C

import numpy as np
import pytest

import terawarp_b200 as tw
from terawarp_b200 import synth

torch = pytest.importorskip("torch")

MATRICES = {
    "identity": lambda d: np.eye(4),
    "shift": lambda d: np.array([[1, 0, 0, -3.0], [0, 1, 0, 5], [0, 0, 1, 2], [0, 0, 0, 1]]),
    "affine": lambda d: synth.random_affine(3, d),
    "rotation": lambda d: synth.random_affine(4, d, rot_deg=60.0, trans=3.0),
    "quarter": lambda d: tw.make_affine(1, 0, (0, 0, 90), d),
    "stretch": lambda d: np.diag([0.2, 2.5, 1.7, 1.0]),
    "too_wide": lambda d: np.diag([9.0, 0.1, 9.0, 1.0]),
    "flat": lambda d: np.diag([1.0, 0.0, 1.0, 1.0]),
}


@pytest.mark.gpu
@pytest.mark.parametrize("dims", [(64, 48, 40), (97, 61, 35), (31, 7, 3), (1, 1, 1), (260, 33, 17)])
@pytest.mark.parametrize("dtype", [np.uint8, np.uint16])
@pytest.mark.parametrize("kind", list(MATRICES))
def test_staged_equals_gathered(ctx, dims, dtype, kind):
    x, y, z = dims
    hook = ctx.lib.tw_internal_set_resample_staging
    hook.restype, hook.argtypes = C.c_int, [C.c_void_p, C.c_int]
    img = np.random.default_rng(x).integers(0, 256 if dtype == np.uint8 else 65536, (z, y, x)).astype(dtype)
    src = torch.from_numpy(img).cuda()
    M = MATRICES[kind](dims)
    for shape in ((z, y, x), (z + 5, max(1, y - 3), x + 21)):
        outs = []
        for on in (1, 0):
            hook(ctx.handle, on)
            dst = torch.from_numpy(np.full(shape, 77, dtype)).cuda()
            torch.cuda.synchronize()
            tw.warp_affine_device(ctx, M, src, dst)
            outs.append(dst.cpu().numpy())
        hook(ctx.handle, 1)
        np.testing.assert_array_equal(outs[0], outs[1])


@pytest.mark.gpu
def test_source_off_a_16_byte_boundary(ctx):
    # such a source is gathered; its neighbours in memory must not be read as part of it
    buf = torch.arange(40 * 50 * 60 + 3, device="cuda").remainder(251).to(torch.uint8)
    view = buf[3:].view(40, 50, 60)
    own = view.clone()
    M = synth.random_affine(1, (60, 50, 40))
    a, b = torch.empty_like(own), torch.empty_like(own)
    torch.cuda.synchronize()
    tw.warp_affine_device(ctx, M, view, a)
    tw.warp_affine_device(ctx, M, own, b)
    np.testing.assert_array_equal(a.cpu().numpy(), b.cpu().numpy())
