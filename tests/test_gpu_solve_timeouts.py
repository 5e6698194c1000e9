"""The landmark solve's bounded waits at limits that run out in different parts
of it -- the factorisation, its hand-overs, the back substitution -- on systems
of two to 21 tiles: the call either reports the time-out or returns the
coefficients, and the context's next solve returns them."""
import ctypes as C

import numpy as np
import pytest

import terawarp_b200 as tw
from terawarp_b200 import synth
from terawarp_b200._lib import TW_ERR_TIMEOUT

pytest.importorskip("torch")


@pytest.mark.gpu
@pytest.mark.parametrize("n", [69, 300, 1345])
def test_solve_recovers_from_time_outs(n):
    sub, tar = synth.lattice_landmarks((700, 600, 300), n, n)
    with tw.Context(0) as c:
        hook = c.lib.tw_internal_set_solve_barrier_ns
        hook.restype, hook.argtypes = C.c_ulonglong, [C.c_void_p, C.c_ulonglong]

        def solve():
            t = tw.tps_solve(c, tar, sub)
            try:
                return t.coeffs()
            finally:
                t.close()

        want = solve()
        for limit_us in (1, 5, 20, 60, 100, 150, 250, 400):
            for _ in range(3):
                hook(c.handle, 1000 * limit_us)
                try:
                    got = solve()
                except tw.TeraWarpError as e:
                    assert e.status == TW_ERR_TIMEOUT
                    hook(c.handle, 0)
                    got = solve()
                for a, b in zip(got, want):
                    np.testing.assert_array_equal(a, b)
