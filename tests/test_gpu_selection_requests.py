"""Trees whose 2:1 balance opens thousands of coarse cells in a sweep (tight groups of particles in
empty space): the order of the requests against the oracle, cell for cell, on both sides of the
4096 requests up to which each request counts the others, with one to three sorted chunks, on
grids of one block and more."""
import numpy as np
import pytest

from apcloud import binding, ics

pytestmark = pytest.mark.gpu


def _groups(k, per, seed):
    rng = np.random.default_rng(seed)
    c = rng.random((3, k)).repeat(per, axis=1)
    x = np.clip(c + 1e-4 * (rng.random(c.shape) - 0.5), 0.0, 1.0 - 1e-9)
    z = np.zeros(k * per)
    return ics.Particles(x[0].copy(), x[1].copy(), x[2].copy(), z.copy(), z.copy(), z.copy())


@pytest.mark.parametrize("groups,per", [(100, 3), (300, 4), (300, 40), (520, 2), (800, 8)])
def test_cells_match_oracle(gpu_lib, oracle_lib, groups, per):
    import refbind

    parts = _groups(groups, per, groups + per)
    g = binding.GpuPath(parts, 21, 1e-9)
    o = refbind.CpuPath("oracle", parts, 21, 1e-9)
    o.set_maxnc(999999)
    try:
        for _ in range(2):  # the second selection finds the tables as the first left them
            m = g.select()
        assert m == o.select()
        cg, co = g.cells(), o.cells()
        assert (cg.nc, cg.nv) == (co.nc, co.nv)
        for f in ("x", "y", "z", "h", "count", "type", "numneigh", "neigh24"):
            assert np.array_equal(getattr(cg, f), getattr(co, f)), f
        nz = co.count > 0
        assert np.array_equal(cg.first[nz], co.first[nz])
    finally:
        o.close()
    g.close()
