"""The V-cycle on a cluster gives the same bits on every run: a block that runs ahead must not
overwrite what a slower one still reads.  The same solve repeated, alone and as many equal boxes
that compete for the SMs, with hierarchies that have one level spread over the cluster above
levels that every block holds whole (that shape has no barrier between the restriction and the
way up but the one this checks), at every sweep parity, as one kernel and as a graph."""
import numpy as np
import pytest

from apcloud import binding, ics

pytestmark = pytest.mark.gpu

PREC = {"mixed": binding.APC_PREC_MIXED, "fp64mg": binding.APC_PREC_FP64_MULTIGRID,
        "vcycle32": binding.APC_PREC_MIXED_VCYCLE}


def _box(n):
    c = 8.0 ** (5.0 / 3.0) * (n / (4.0 / 3.0 * np.pi * 0.3 ** 3)) ** (-2.0 / 3.0)
    return ics.uniform_ball(n, 0.3, seed=3), c


@pytest.mark.parametrize("sweeps", [1, 2, 3])
@pytest.mark.parametrize("precision", sorted(PREC))
@pytest.mark.parametrize("n", [1500, 6000, 60000])
def test_same_bits_on_every_run(gpu_lib, n, precision, sweeps):
    parts, c = _box(n)
    kw = dict(precision=PREC[precision], mg_sweeps=sweeps)
    g = binding.GpuPath(parts, 21, c, **kw)
    g.select()
    first = None
    for _ in range(8):
        g.solve(1.0 / n, 30.0, -1.0)
        got = (g.solve_stats()["potential_its"], g.fields().potential)
        first = first or got
        assert got[0] == first[0] and np.array_equal(got[1], first[1])
    g.close()
    b = binding.BatchPath([(parts, dict(depth=21, gfd_c=c, **kw))] * 8)
    b.step([(0.0, 1.0 / n, 30.0, -1.0, 0.0, 0.0)] * 8)
    for box in b.boxes:
        assert box.solve_stats()["potential_its"] == first[0]
        assert np.array_equal(box.fields().potential, first[1])
    b.close()
