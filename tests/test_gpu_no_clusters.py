"""On a device without clusters of 16 blocks the multigrid solves run in the forms without them:
one small system (one level), whole hierarchies that a cluster would hold, grid levels above
them.  The residual is formed here in FP64 from the assembled matrix, with the bound of the
cluster form's test: 1e-10 of the stopping test and 5 % for another order of the sums."""
import numpy as np
import pytest

from apcloud import binding, ics

pytestmark = pytest.mark.gpu

C_POT = 30.0
PREC = {"mixed": binding.APC_PREC_MIXED, "fp64mg": binding.APC_PREC_FP64_MULTIGRID,
        "vcycle32": binding.APC_PREC_MIXED_VCYCLE}


def _box(name):
    if name.startswith("ball"):
        n = int(name[4:])
        return ics.uniform_ball(n, 0.3, seed=3), 8.0 ** (5.0 / 3.0) * (n / (4.0 / 3.0 * np.pi * 0.3 ** 3)) ** (-2.0 / 3.0)
    side = int(name[3:])
    c = 2e-2 if side == 4 else 1.28 * 8.0 ** (5.0 / 3.0) * side ** -2.0
    return ics.zeldovich(side, -2.0, 0.25, 0.05, 1.0, 0.0, seed=4), c


@pytest.mark.parametrize("precision", sorted(PREC))
@pytest.mark.parametrize("name", ["zel4", "zel17", "ball1500", "ball60011"])
def test_solves_without_clusters(gpu_lib, name, precision):
    parts, c = _box(name)
    lib = binding.load_library(gpu_lib)
    out = []
    for off in (0, 1):
        g = binding.GpuPath(parts, 21, c, precision=PREC[precision])
        lib.apc_test_no_clusters(g.h, off)
        g.select()
        g.solve(1.0 / parts.n, C_POT, -1.0)
        out.append((g.solve_stats(), g.fields(), g.kernel_launches()))
        cells, (ptr, col, val) = g.cells(), g.matrix(1)
        g.close()
    (s0, _, l0), (s, f, l1) = out
    assert l1 != l0  # another form ran
    m = cells.m
    row = np.repeat(np.arange(m), np.diff(ptr))
    v = cells.h[:m] ** 3
    b = (f.density - np.sum(f.density * v) / np.sum(v)) * C_POT
    ax = np.bincount(row, weights=val * f.potential[col], minlength=m)
    d = np.zeros(m)
    d[row[row == col]] = val[row == col]
    d[d == 0.0] = 1.0
    bn = np.linalg.norm(b / d)
    assert s["density_reason"] in (2, 3) and s["potential_reason"] in (2, 3)
    if bn > 1e-12 * C_POT / np.abs(d).max():  # equal densities: the right-hand side is rounding alone
        assert np.linalg.norm((b - ax) / d) <= 1.05e-10 * bn
        # the same operator in other code: rounding moves the count by at most two
        assert precision == "mixed" or abs(s["potential_its"] - s0["potential_its"]) <= 2
