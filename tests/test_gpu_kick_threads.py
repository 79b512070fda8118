"""apc_move_velocity_noalloc keeps nothing between calls, and a device takes one call at a time:
host threads that call it, on one stream or each on its own, get the largest change, the outputs
or the refusal of their own call."""
import ctypes as C
import threading

import numpy as np
import pytest

from apcloud import binding

pytestmark = pytest.mark.gpu

DT, CV, CALLS = 0.01, 1.7, 60


@pytest.mark.parametrize("shared", [True, False])
def test_host_threads(gpu_lib, shared):
    import torch

    lib = binding.load_library()
    dev = lambda a, t=torch.float64: torch.as_tensor(np.ascontiguousarray(a), dtype=t, device="cuda")  # noqa: E731
    jobs = []
    for k in range(4):
        rng = np.random.default_rng(k)
        n = 20000 * (k + 1) + 7
        m = n // 9
        count = rng.multinomial(n, np.ones(m) / m)
        first = np.cumsum(count) - count
        cell = np.repeat(np.arange(m), count)
        if k == 3:  # this thread's ranges leave a particle out
            count[np.argmax(count)] -= 1
        cen, der = rng.random((3, m)), (k + 1.0) * rng.standard_normal((m, 9))
        x = rng.random((3, n))
        d, (px, py, pz) = der[cell], x - cen[:, cell]
        a = [((d[:, 0] + px * d[:, 3]) + py * d[:, 6]) + pz * d[:, 7],
             ((d[:, 1] + px * d[:, 6]) + py * d[:, 4]) + pz * d[:, 8],
             ((d[:, 2] + px * d[:, 7]) + py * d[:, 8]) + pz * d[:, 5]]
        sq = (a[0] * a[0] + a[1] * a[1]) + a[2] * a[2]
        jobs.append(dict(n=n, m=m, ranges=[dev(first, torch.int32), dev(count, torch.int32)],
                         arrs=[dev(c) for c in cen] + [dev(der)] + [dev(q) for q in x], a=a,
                         v=[dev(np.zeros(n)) for _ in range(3)], acc=[dev(np.zeros(n)) for _ in range(3)],
                         want=np.sqrt(np.max((((sq * CV) * CV) * DT) * DT)), got=[]))
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in jobs]

    def work(j, stream):
        for _ in range(CALLS):
            dv = C.c_double(-1.0)
            rc = lib.apc_move_velocity_noalloc(j["n"], j["m"], *[t.data_ptr() for t in j["ranges"] + j["arrs"]],
                                               *[t.data_ptr() for t in j["v"] + j["acc"]], DT, CV, C.byref(dv),
                                               stream.cuda_stream)
            j["got"].append((rc, dv.value))

    threads = [threading.Thread(target=work, args=(j, streams[0 if shared else k])) for k, j in enumerate(jobs)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k, j in enumerate(jobs):
        assert j["got"] == [(-1, -1.0) if k == 3 else (0, j["want"])] * CALLS, k
        for q in range(3):
            v = np.zeros(j["n"])
            for _ in range(CALLS if k < 3 else 0):
                v = v + (j["a"][q] * CV) * DT
            assert np.array_equal(j["v"][q].cpu().numpy(), v), (k, q)
