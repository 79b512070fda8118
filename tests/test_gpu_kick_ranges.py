"""apc_move_velocity_noalloc over the shapes its cells may have - one cell of everything, cells of
thousands beside cells of one, empty cells, ranges in any order - against NumPy, which rounds
each product and sum as the kernel does (equality), and its refusals: ranges that overlap, leave
a hole, run out of bounds or hold too many particles leave every output untouched."""
import ctypes as C

import numpy as np
import pytest

from apcloud import binding

pytestmark = pytest.mark.gpu

DT, CV = 0.01, 1.7


def _counts(kind, n, rng):
    if kind == "one":
        return np.array([n])
    if kind == "ones":
        return np.ones(n, int)
    if kind == "mixed":  # a cell of most particles, some of hundreds, many small, some empty
        c = [n // 2]
        while sum(c) < n:
            c.append(int(min(n - sum(c), rng.choice([0, 1, 3, 9, 70, 300, 2047, 2048, 2500]))))
        return np.array(c)
    c = rng.multinomial(n, np.ones(max(1, n // 12)) / max(1, n // 12))
    return c


def _call(lib, n, first, count, arrs, v, acc):
    dv = C.c_double()
    rc = lib.apc_move_velocity_noalloc(n, len(first), first.data_ptr(), count.data_ptr(), *[a.data_ptr() for a in arrs],
                                       *[a.data_ptr() for a in v], *[a.data_ptr() for a in acc], DT, CV, C.byref(dv),
                                       None)
    return rc, dv.value


@pytest.mark.parametrize("kind,n", [("one", 1), ("one", 5000), ("ones", 33), ("ones", 4097), ("mixed", 30011),
                                    ("even", 7), ("even", 100003), ("mixed", 1 << 20)])
def test_kick_ranges(gpu_lib, kind, n):
    import torch

    rng = np.random.default_rng(n)
    lib = binding.load_library()
    count = _counts(kind, n, rng)
    first = np.cumsum(count) - count
    order = rng.permutation(len(count))  # the cells in any order
    first, count = first[order], count[order]
    m = len(count)
    cen, der = rng.random((3, m)), rng.standard_normal((m, 9))
    x, v0 = rng.random((3, n)), rng.standard_normal((3, n))
    dev = lambda a, t=torch.float64: torch.as_tensor(np.ascontiguousarray(a), dtype=t, device="cuda")  # noqa: E731
    df, dc = dev(first, torch.int32), dev(count, torch.int32)
    arrs = [dev(c) for c in cen] + [dev(der)] + [dev(a) for a in x]
    v, acc = [dev(a) for a in v0], [torch.full((n,), 7.0, dtype=torch.float64, device="cuda") for _ in range(3)]
    torch.cuda.synchronize()
    cell = np.empty(n, int)
    for i in np.nonzero(count)[0]:
        cell[first[i]:first[i] + count[i]] = i
    d, (px, py, pz) = der[cell], x - cen[:, cell]
    a = [((d[:, 0] + px * d[:, 3]) + py * d[:, 6]) + pz * d[:, 7],
         ((d[:, 1] + px * d[:, 6]) + py * d[:, 4]) + pz * d[:, 8],
         ((d[:, 2] + px * d[:, 7]) + py * d[:, 8]) + pz * d[:, 5]]
    for k in range(2):  # the second call finds the scratch as the first left it
        rc, dv = _call(lib, n, df, dc, arrs, v, acc)
        assert rc == 0
        sq = (a[0] * a[0] + a[1] * a[1]) + a[2] * a[2]
        assert dv == np.sqrt(np.max((((sq * CV) * CV) * DT) * DT))
        for q in range(3):
            v0[q] = v0[q] + (a[q] * CV) * DT
            assert np.array_equal(v[q].cpu().numpy(), v0[q]) and np.array_equal(acc[q].cpu().numpy(), a[q])
    # refusals
    bad = []
    big = int(np.argmax(count))
    for f2, c2 in (((first[big] + 1), count[big]), (first[big], count[big] + 1), (first[big], count[big] - 1),
                   (-1, count[big]), (first[big], -1), (n, 1)):
        f, c = first.copy(), count.copy()
        f[big], c[big] = f2, c2
        bad.append((f, c))
    if m > 1 and n > 1:  # two cells swap places: n particles in all, an overlap and a hole
        f = first.copy()
        nz = np.nonzero(count)[0]
        if len(nz) > 1 and count[nz[0]] != count[nz[1]]:
            f[nz[0]], f[nz[1]] = first[nz[1]], first[nz[0]]
            bad.append((f, count.copy()))
    for f, c in bad:
        rc, _ = _call(lib, n, dev(f, torch.int32), dev(c, torch.int32), arrs, v, acc)
        assert rc == -1
        for q in range(3):
            assert np.array_equal(v[q].cpu().numpy(), v0[q]) and np.array_equal(acc[q].cpu().numpy(), a[q])
    assert _call(lib, n, df, dc, arrs, v, acc)[0] == 0
