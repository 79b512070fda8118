"""The multigrid aggregation kernel, through the solves that use it: the number of levels is the
one that counting distinct parent codes gives, from boxes of one level to boxes of a million
cells, and with more cells than the first box of the context (its buffers grow)."""
import numpy as np
import pytest

from apcloud import binding, ics

pytestmark = pytest.mark.gpu


def _levels(codes):
    n = 1
    while len(codes) > 64:
        parents = np.unique(np.where(codes > 1, codes >> np.uint64(3), np.uint64(1)))
        if len(parents) >= len(codes):
            break
        codes = parents
        n += 1
    return n


@pytest.mark.parametrize("kind,size,gfd_c", [("zel", 4, 2e-2), ("ball", 300, 1e-1), ("ball", 3001, 2e-3),
                                             ("zel", 30, 1e-3), ("clump", 60000, 5e-3), ("zel", 100, 1.5e-4)])
def test_levels_and_convergence(gpu_lib, kind, size, gfd_c):
    g = None
    for seed in (1, 2):
        if kind == "zel":
            parts = ics.zeldovich(size, -2.0, 0.2 if seed == 1 else 1.0, 0.05, 1.0, 0.0, seed=seed)
        else:
            parts = ics.uniform_ball(size, 0.3 if seed == 1 else 0.2, seed=seed)
            if kind == "clump":
                parts.x[: size // 2] = 0.5 + 0.01 * (parts.x[: size // 2] - 0.5)
        if g is None:
            g = binding.GpuPath(parts, 21, gfd_c, precision=binding.APC_PREC_MIXED_VCYCLE)
        else:
            g.set_particles(parts)
        g.select()
        g.solve(1.0 / parts.n, 30.0, -1.0)
        st = g.solve_stats()
        assert st["potential_reason"] in (2, 3) and st["density_reason"] in (2, 3)
        assert st["mg_levels"] == _levels(g.codes())
    g.close()
