"""Operator calls on device-resident volumes: one launch over the volume, or
slab by slab when that launch's workspace is over the context's budget."""
import numpy as np
import pytest

import terawarp_b200 as tw
from terawarp_b200 import synth

torch = pytest.importorskip("torch")


@pytest.mark.gpu
def test_device_volume_falls_back_to_slabs_within_the_budget(ctx):
    x, y, z, g, n = 1024, 1024, 256, 16, 8
    sub, tar = synth.lattice_landmarks((x, y, z), n, 4)
    src = torch.randint(0, 256, (z, y, x), dtype=torch.uint8, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    torch.cuda.synchronize()
    want = tw.imgwarp_smallmemory_image(ctx, sub, tar, g, g, g, 1, 0, src)
    nodes = 16 * tw.grid_size(x, g) * tw.grid_size(y, g) * tw.grid_size(z, g)
    # the node grid, and a workspace of at most 250,000 bytes: the whole
    # volume's 4096 work units take 80 bytes each, a slab's 2048 fit
    with tw.Context(0, nodes + 4096 + 250_000) as small:
        got = tw.imgwarp_smallmemory_image(small, sub, tar, g, g, g, 1, 0, src)
        np.testing.assert_array_equal(got.cpu().numpy(), want.cpu().numpy())
        assert small.kernel_launches > 30  # several slabs


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [np.uint8, np.uint16])
def test_device_volume_equals_host_volume(ctx, dtype):
    x, y, z, g = 700, 523, 150, 8
    sub, tar = synth.lattice_landmarks((x, y, z), 40, 5)
    img = np.random.default_rng(2).integers(0, 256 if dtype == np.uint8 else 4096, (z, y, x)).astype(dtype)
    dev = torch.from_numpy(img).cuda()
    torch.cuda.synchronize()
    a = tw.imgwarp_smallmemory_image(ctx, sub, tar, g, g, g, 1, 0, img)
    b = tw.imgwarp_smallmemory_image(ctx, sub, tar, g, g, g, 1, 0, dev)
    np.testing.assert_array_equal(a, b.cpu().numpy())
