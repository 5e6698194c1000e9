"""Calls from several threads, each with a context of its own."""
import threading

import numpy as np
import pytest

import terawarp_b200 as tw

torch = pytest.importorskip("torch")


@pytest.mark.gpu
def test_affine_calls_of_different_boxes_in_parallel(ctx):
    # each thread's tiles are staged in boxes of another size, so each launch
    # asks for another amount of shared memory
    src = torch.randint(0, 256, (48, 64, 96), dtype=torch.uint8, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    mats = [np.diag([s, 1.0, r, 1.0]) for s, r in ((1.0, 1.0), (1.0, 1.4), (1.4, 1.0), (0.5, 0.5), (1.2, 1.2), (0.8, 0.6))]
    want = []
    for M in mats:
        dst = torch.empty_like(src)
        tw.warp_affine_device(ctx, M, src, dst)
        want.append(dst)
    errors = []

    def work(M, ref):
        try:
            with tw.Context(0) as c:
                dst = torch.empty_like(src)
                torch.cuda.synchronize()
                for _ in range(600):
                    tw.warp_affine_device(c, M, src, dst)
                if not torch.equal(dst, ref):
                    errors.append(f"{np.diag(M)}: other voxels")
        except Exception as e:  # noqa: BLE001
            errors.append(f"{np.diag(M)}: {e}")

    threads = [threading.Thread(target=work, args=a) for a in zip(mats, want)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
