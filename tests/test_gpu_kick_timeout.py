"""apc_move_velocity_noalloc with a wait that gives up: the call kicks every particle or none.  The
first block's wait runs out after a few polls while the warp that marks a wide cell is still at
work in a later block, which then finds every block arrived."""
import ctypes as C

import numpy as np
import pytest

from apcloud import binding

pytestmark = pytest.mark.gpu

DT, CV = 0.01, 1.7
TIMEOUT = -10


def test_all_or_nothing(gpu_lib):
    import torch

    lib = binding.load_library(gpu_lib)
    call = lib.apc_test_move_velocity_noalloc
    call.restype = C.c_int
    call.argtypes = [C.c_int, C.c_int, C.c_int] + [C.c_void_p] * 15 + [C.c_double, C.c_double, C.c_void_p, C.c_void_p]
    n, seen = 1 << 20, set()
    dev = lambda a, t=torch.float64: torch.as_tensor(np.ascontiguousarray(a), dtype=t, device="cuda")  # noqa: E731
    for wide in (n - 20000, n // 2, n // 16, 3000, 300, 10):
        rest = n - wide  # cells of 10, the wide one last
        count = np.concatenate([np.full(rest // 10, 10), [rest % 10, wide]])
        first, m = np.cumsum(count) - count, len(count)
        rng = np.random.default_rng(wide)
        arrs = [dev(rng.random(m)) for _ in range(3)] + [dev(rng.standard_normal((m, 9)))]
        arrs += [dev(rng.random(n)) for _ in range(3)]
        df, dc = dev(first, torch.int32), dev(count, torch.int32)
        v0 = dev(rng.standard_normal((3, n)))

        def kick(limit):
            v, acc = v0.clone(), torch.full((3, n), 7.0, dtype=torch.float64, device="cuda")
            torch.cuda.synchronize()
            rc = call(limit, n, m, df.data_ptr(), dc.data_ptr(), *[a.data_ptr() for a in arrs],
                      *[a.data_ptr() for a in (*v, *acc)], DT, CV, None, None)
            return rc, v, acc

        rc, v1, acc1 = kick(1 << 21)
        assert rc == 0
        for limit in (1, 2, 3, 5, 8, 20, 60, 200):
            for _ in range(5):
                rc, v, acc = kick(limit)
                seen.add(rc)
                if rc == 0:
                    assert torch.equal(v, v1) and torch.equal(acc, acc1), (wide, limit)
                else:
                    assert rc == TIMEOUT
                    assert torch.equal(v, v0) and bool((acc == 7.0).all()), (wide, limit)
    assert seen == {0, TIMEOUT}
