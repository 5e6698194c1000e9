"""A host volume warped slab by slab is uploaded while its first slabs are
resampled: no launch may read all of the source (a ragged one is not copied into
padded rows then, however large the slab)."""
import ctypes as C

import numpy as np
import pytest

import terawarp_b200 as tw
from terawarp_b200 import synth

torch = pytest.importorskip("torch")


@pytest.mark.gpu
def test_ragged_source_is_not_copied_while_it_arrives(ctx):
    # two slabs of 16 planes, 64 M voxels each
    x, y, z, g = 2003, 2003, 32, 16
    hook = ctx.lib.tw_internal_set_resample_staging
    hook.restype, hook.argtypes = C.c_int, [C.c_void_p, C.c_int]
    sub, tar = synth.lattice_landmarks((x, y, z), 20, 4)
    src = torch.randint(0, 256, (z, y, x), dtype=torch.uint8, generator=torch.Generator().manual_seed(1)).pin_memory()
    outs, launches = [], []
    for on in (1, 0):
        hook(ctx.handle, on)
        before = ctx.kernel_launches
        outs.append(tw.imgwarp_smallmemory_image(ctx, tar, sub, g, g, g, 1, 0, src).clone())
        launches.append(ctx.kernel_launches - before)
    hook(ctx.handle, 1)
    assert launches[0] == launches[1]  # one gathered launch per slab either way
    # resident on the device the same volume is copied and staged
    dev = src.cuda()
    torch.cuda.synchronize()
    before = ctx.kernel_launches
    out = tw.imgwarp_smallmemory_image(ctx, tar, sub, g, g, g, 1, 0, dev)
    assert ctx.kernel_launches - before > launches[0]
    np.testing.assert_array_equal(outs[0].numpy(), outs[1].numpy())
    np.testing.assert_array_equal(outs[0].numpy(), out.cpu().numpy())
