"""A kernel that gave up waiting: the next call that waits for the context's
stream reports it, once, and the context goes on."""
import ctypes as C

import numpy as np
import pytest

import terawarp_b200 as tw
from terawarp_b200._lib import TW_ERR_TIMEOUT

torch = pytest.importorskip("torch")


@pytest.mark.gpu
@pytest.mark.parametrize("call", ["affine", "tps", "operator", "synchronize"])
def test_reported_once(call):
    src = torch.randint(0, 256, (40, 48, 64), dtype=torch.uint8, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    dst = torch.empty_like(src)
    nodes = torch.zeros(tuple(tw.grid_size(n, 16) for n in src.shape) + (4,), dtype=torch.float32, device="cuda")
    M = np.diag([1.1, 0.9, 1.0, 1.0])
    pts = np.random.default_rng(2).uniform(3, 36, (20, 3)).astype(np.float32)
    torch.cuda.synchronize()
    with tw.Context(0) as c, tw.Context(0) as other:
        raise_error = c.lib.tw_internal_raise_kernel_error
        raise_error.restype, raise_error.argtypes = C.c_int, [C.c_void_p]

        def run(ctx):
            if call == "affine":
                tw.warp_affine_device(ctx, M, src, dst)
            elif call == "tps":
                tw.warp_tps_device(ctx, nodes, 16, src, dst)
            elif call == "operator":
                tw.q_imagewarp_affine_image(ctx, pts, pts + 0.5, src, out=dst)
            else:
                ctx.synchronize()
            return dst.cpu().numpy()

        want = run(c)
        assert raise_error(c.handle) == 0
        with pytest.raises(tw.TeraWarpError) as e:
            run(c)
        assert e.value.status == TW_ERR_TIMEOUT
        np.testing.assert_array_equal(run(c), want)
        assert raise_error(c.handle) == 0
        run(other)  # another context's word
        with pytest.raises(tw.TeraWarpError):
            run(c)
        run(c)
