"""apc_move_velocity_noalloc where cells are kicked piece by piece (256 particles and more) beside
cells that are not: counts on both sides of the line and of whole pieces (128), as many such
cells as can be, and mean counts on both sides of every change of the lanes per cell.  Against
NumPy, which rounds each product and sum as the kernel does (equality)."""
import ctypes as C

import numpy as np
import pytest

from apcloud import binding

pytestmark = pytest.mark.gpu

DT, CV = 0.01, 1.7


@pytest.mark.parametrize("counts", [[255], [256], [257, 255, 0, 256, 384, 385, 511, 512, 513, 1],
                                    [256] * 4096, [257] * 300 + [255] * 300, [8] * 700, [9] + [8] * 700,
                                    [16] * 500, [17] + [16] * 500, [33] + [32] * 500, [32] * 500, [64] * 300,
                                    [65] + [64] * 300, [128] * 50, [100000] * 3 + [1] * 5000, [1] * 5000 + [100000]],
                         ids=lambda c: "%dx%d" % (len(c), max(c)))
def test_pieces(gpu_lib, counts):
    import torch

    lib = binding.load_library(gpu_lib)
    count = np.array(counts)
    n, m = int(count.sum()), len(counts)
    rng = np.random.default_rng(n)
    first = np.cumsum(count) - count
    cell = np.repeat(np.arange(m), count)
    cen, der = rng.random((3, m)), rng.standard_normal((m, 9))
    x, v0 = rng.random((3, n)), rng.standard_normal((3, n))
    dev = lambda a, t=torch.float64: torch.as_tensor(np.ascontiguousarray(a), dtype=t, device="cuda")  # noqa: E731
    arrs = [dev(c) for c in cen] + [dev(der)] + [dev(a) for a in x]
    v, acc = [dev(a) for a in v0], [torch.zeros(n, dtype=torch.float64, device="cuda") for _ in range(3)]
    df = dev(first, torch.int32)
    torch.cuda.synchronize()

    def kick(c):
        dv, dc = C.c_double(), dev(c, torch.int32)
        torch.cuda.synchronize()
        rc = lib.apc_move_velocity_noalloc(n, m, df.data_ptr(), dc.data_ptr(), *[a.data_ptr() for a in arrs],
                                           *[a.data_ptr() for a in v], *[a.data_ptr() for a in acc], DT, CV,
                                           C.byref(dv), None)
        return rc, dv.value

    j = int(np.argmax(count))
    if j + 2 < m and count[j + 1] > 0 and count[j] > 1:
        # n in all, but the largest cell's second-last particle is the last of its range and the
        # next cell's range runs one too far: a hole before it, and an overlap after it
        bad = count.copy()
        bad[j] -= 1
        bad[j + 1] += 1
        assert kick(bad)[0] == -1
        assert all(np.array_equal(v[q].cpu().numpy(), v0[q]) for q in range(3))
    rc, dv = kick(count)
    assert rc == 0
    d, (px, py, pz) = der[cell], x - cen[:, cell]
    a = [((d[:, 0] + px * d[:, 3]) + py * d[:, 6]) + pz * d[:, 7],
         ((d[:, 1] + px * d[:, 6]) + py * d[:, 4]) + pz * d[:, 8],
         ((d[:, 2] + px * d[:, 7]) + py * d[:, 8]) + pz * d[:, 5]]
    for q in range(3):
        assert np.array_equal(acc[q].cpu().numpy(), a[q])
        assert np.array_equal(v[q].cpu().numpy(), v0[q] + (a[q] * CV) * DT)
    sq = (a[0] * a[0] + a[1] * a[1]) + a[2] * a[2]
    assert dv == np.sqrt(np.max((((sq * CV) * CV) * DT) * DT))
