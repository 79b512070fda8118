"""The selection kernel against the oracle, cell for cell in the reference's order: particle
counts around a warp, a block and the whole grid, trees cut by the depth limit, and clumps whose
2:1 balance opens from a handful to thousands of coarse cells per sweep (more than one tile of
the ranking), in one context run twice (the request tables are reused)."""
import numpy as np
import pytest

from apcloud import binding, ics

pytestmark = pytest.mark.gpu


def _parts(kind, n, seed):
    rng = np.random.default_rng(seed)
    x = rng.random((3, n))
    if kind == "clump":  # half of the particles in a few tight groups off the cell corners
        m = n // 2
        centre = rng.random((3, 7))[:, rng.integers(0, 7, m)]
        x[:, :m] = np.mod(centre + 1e-4 * rng.standard_normal((3, m)), 1.0)
    elif kind == "line":  # a thin wall: a deep sheet of cells beside coarse ones
        x[2] = 0.37 + 1e-5 * rng.random(n)
    z = np.zeros(n)
    return ics.Particles(x[0].copy(), x[1].copy(), x[2].copy(), z.copy(), z.copy(), z.copy())


@pytest.mark.parametrize("depth", [21, 6])
@pytest.mark.parametrize("kind,n,gfd_c", [
    ("uniform", 1, 0.1), ("uniform", 7, 0.4), ("uniform", 33, 0.02), ("uniform", 2049, 4e-3),
    ("uniform", 70001, 6e-3), ("clump", 513, 2e-3), ("clump", 9000, 1e-3), ("clump", 150000, 2e-4),
    ("line", 40000, 1e-3)])
def test_cells_match_oracle(gpu_lib, oracle_lib, kind, n, gfd_c, depth):
    import refbind

    g = None
    for seed in (1, 2):
        parts = _parts(kind, n, seed)
        if g is None:
            g = binding.GpuPath(parts, depth, gfd_c)
        else:
            g.set_particles(parts)
        o = refbind.CpuPath("oracle", parts, depth, gfd_c)
        o.set_maxnc(999999)  # the reference gives up at a budget of 1e6 temp nodes
        try:
            assert g.select() == o.select()
            cg, co = g.cells(), o.cells()
            assert (cg.nc, cg.nv) == (co.nc, co.nv)
            for f in ("x", "y", "z", "h", "count", "type", "numneigh", "neigh24"):
                assert np.array_equal(getattr(cg, f), getattr(co, f)), f
            nz = co.count > 0
            assert np.array_equal(cg.first[nz], co.first[nz])
        finally:
            o.close()
    g.close()
