"""apc_move_velocity_noalloc with empty cells whose `first` is any value: nothing is formed from it.
At each number of lanes per cell (it follows the mean count), against NumPy, which rounds each
product and sum as the kernel does (equality)."""
import ctypes as C

import numpy as np
import pytest

from apcloud import binding

pytestmark = pytest.mark.gpu

DT, CV = 0.01, 1.7
INT_MAX = 2 ** 31 - 1


@pytest.mark.parametrize("mean", [1, 6, 12, 24, 200])
@pytest.mark.parametrize("value", [INT_MAX, INT_MAX - 5, -1, -INT_MAX - 1, 1 << 20])
def test_first_of_an_empty_cell_is_not_used(gpu_lib, mean, value):
    import torch

    rng = np.random.default_rng(mean)
    lib = binding.load_library()
    n, m = 3001, max(2, 3001 // mean)
    count = rng.multinomial(n, np.ones(m) / m)
    count[m // 2] += count[0]
    count[0] = 0
    first = np.cumsum(count) - count
    cell = np.repeat(np.arange(m), count)
    first[count == 0] = value
    cen, der = rng.random((3, m)), rng.standard_normal((m, 9))
    x, v0 = rng.random((3, n)), rng.standard_normal((3, n))
    dev = lambda a, t=torch.float64: torch.as_tensor(np.ascontiguousarray(a), dtype=t, device="cuda")  # noqa: E731
    df, dc = dev(first, torch.int32), dev(count, torch.int32)
    arrs = [dev(c) for c in cen] + [dev(der)] + [dev(a) for a in x]
    v, acc = [dev(a) for a in v0], [torch.zeros(n, dtype=torch.float64, device="cuda") for _ in range(3)]
    torch.cuda.synchronize()
    dv = C.c_double()
    rc = lib.apc_move_velocity_noalloc(n, m, df.data_ptr(), dc.data_ptr(), *[a.data_ptr() for a in arrs],
                                       *[a.data_ptr() for a in v], *[a.data_ptr() for a in acc], DT, CV, C.byref(dv),
                                       None)
    assert rc == 0
    d, (px, py, pz) = der[cell], x - cen[:, cell]
    a = [((d[:, 0] + px * d[:, 3]) + py * d[:, 6]) + pz * d[:, 7],
         ((d[:, 1] + px * d[:, 6]) + py * d[:, 4]) + pz * d[:, 8],
         ((d[:, 2] + px * d[:, 7]) + py * d[:, 8]) + pz * d[:, 5]]
    for q in range(3):
        assert np.array_equal(acc[q].cpu().numpy(), a[q])
        assert np.array_equal(v[q].cpu().numpy(), v0[q] + (a[q] * CV) * DT)
    sq = (a[0] * a[0] + a[1] * a[1]) + a[2] * a[2]
    assert dv.value == np.sqrt(np.max((((sq * CV) * CV) * DT) * DT))
