"""Calls that go on without a workspace that is over the context's budget -- a
gathered launch in place of a staged one, a source that is not copied, slabs in
place of one launch -- succeed and leave no error text behind."""
import numpy as np
import pytest

import terawarp_b200 as tw
from terawarp_b200 import synth

torch = pytest.importorskip("torch")


def _text(ctx):
    return (ctx.lib.tw_ctx_last_error(ctx.handle) or b"").decode()


@pytest.mark.gpu
@pytest.mark.parametrize("dims,interp", [((256, 256, 264), 1), ((515, 401, 250), 0)])
def test_launch_without_its_workspace(ctx, dims, interp):
    g = 16
    src = torch.randint(0, 256, dims[::-1], dtype=torch.uint8, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    nodes = torch.from_numpy(np.random.default_rng(1).normal(0, 1, tuple(tw.grid_size(n, g) for n in dims[::-1]) + (4,)).astype(np.float32)).cuda()
    want, got = torch.empty_like(src), torch.empty_like(src)
    torch.cuda.synchronize()
    tw.warp_tps_device(ctx, nodes, g, src, want, interp=interp)
    with tw.Context(0, 4096) as small:  # no room for plans or copies
        before = small.kernel_launches
        tw.warp_tps_device(small, nodes, g, src, got, interp=interp)
        assert small.kernel_launches - before == 1
        assert _text(small) == ""
        # an earlier failure's text stays
        with pytest.raises(tw.TeraWarpError):
            tw.warp_tps_device(small, nodes, 5, src, got)
        said = _text(small)
        tw.warp_tps_device(small, nodes, g, src, got, interp=interp)
        assert said and _text(small) == said
    np.testing.assert_array_equal(got.cpu().numpy(), want.cpu().numpy())


@pytest.mark.gpu
def test_volume_in_slabs():
    x, y, z, g, n = 1024, 1024, 256, 16, 8
    sub, tar = synth.lattice_landmarks((x, y, z), n, 4)
    src = torch.zeros((z, y, x), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    nodes = 16 * tw.grid_size(x, g) * tw.grid_size(y, g) * tw.grid_size(z, g)
    with tw.Context(0, nodes + 4096 + 250_000) as small:  # room for a slab's plans, not for the volume's
        tw.imgwarp_smallmemory_image(small, sub, tar, g, g, g, 1, 0, src)
        assert small.kernel_launches > 30
        assert _text(small) == ""
