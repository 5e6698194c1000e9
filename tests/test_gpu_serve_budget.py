"""The server's workspaces stay within its budget: a ragged source is copied into
padded rows only where the copy fits."""
import numpy as np
import pytest

import terawarp_b200 as tw
from terawarp_b200 import synth
from terawarp_b200.api import Server

torch = pytest.importorskip("torch")


@pytest.mark.gpu
@pytest.mark.parametrize("budget_mb,copies", [(64, False), (512, True)])
def test_padded_copies_fit_the_budget(ctx, budget_mb, copies):
    x, y, z, g = 515, 401, 250, 16  # 51.6 M voxels of uint16: a copy of 104 MB
    sub, tar = synth.lattice_landmarks((x, y, z), 20, 4)
    src = torch.randint(0, 256, (z, y, x), dtype=torch.int32, device="cuda", generator=torch.Generator("cuda").manual_seed(1)).to(torch.uint16)
    dst = torch.empty_like(src)
    tiny = torch.zeros((64, 64, 64), dtype=torch.uint16, device="cuda")
    tiny_out = torch.empty_like(tiny)
    want = tw.imgwarp_smallmemory_image(ctx, tar, sub, g, g, g, 1, 0, src)
    torch.cuda.synchronize()
    s = Server(ctx, hbm_budget_bytes=budget_mb << 20)
    try:
        s.wait(s.submit_tps(sub, tar, g, tiny, tiny_out))
        free = torch.cuda.mem_get_info()[0]
        s.wait(s.submit_tps(sub, tar, g, src, dst))
        taken = (free - torch.cuda.mem_get_info()[0]) / 2**20  # (the server's pool keeps its blocks)
    finally:
        s.close()
    assert taken <= budget_mb
    assert (taken > 90) == copies
    np.testing.assert_array_equal(dst.cpu().numpy(), want.cpu().numpy())
