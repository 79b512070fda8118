"""The particle -> cell map of the kick over cells of every size it treats apart: none, up to 8
and up to 64 particles, more than 64 (the whole warp on one cell), and a cell count that is no
multiple of 32.  Given the fields, the accelerations are the interpolation's own operations, so
the comparison is bit for bit."""
import numpy as np
import pytest

from apcloud import binding, ics


def particles(seed, cluster):
    """A uniform background, and clusters that end in cells of the smallest size."""
    rng = np.random.default_rng(seed)
    side = 16
    g = (np.arange(side) + 0.5) / side
    pts = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    pts = pts + (rng.random(pts.shape) - 0.5) * 0.6 / side
    own = [(0.3 + 0.02 * k + 0.01 * rng.random((c, 3))) for k, c in enumerate(cluster)]
    x = np.concatenate([pts, *own])
    v = np.zeros(len(x))
    return ics.Particles(*(np.ascontiguousarray(a) for a in x.T), v, v.copy(), v.copy())


SIZES = [(3, (7, 8, 9)), (5, (63, 64, 65, 129)), (8, (5000, 20, 1000))]
DEPTH, GFD_C = 5, 5e-3  # 4,110 cells


@pytest.mark.gpu
@pytest.mark.parametrize("seed,cluster", SIZES)
def test_kick_takes_each_particle_from_its_cell(gpu_lib, seed, cluster):
    gp = binding.GpuPath(particles(seed, cluster), DEPTH, GFD_C, precision=binding.APC_PREC_MIXED)
    try:
        gp.select()
        gp.solve(1.0, -1.0)
        gp.move_velocity(0.01, 1.0)
        c, d = gp.cells(), gp.fields().deriv
        order = gp.keys()[1]  # the cells' ranges count particles in key order
        x, y, z, _, _, _, ax, ay, az = (p[order] for p in gp.particles())
        assert c.m % 32 and c.count.max() >= max(cluster) // 8
        s = np.concatenate([np.arange(f, f + k) for f, k in zip(c.first, c.count)])
        i = np.repeat(np.arange(c.m), c.count)
        assert np.array_equal(np.sort(s), np.arange(x.size))
        dx, dy, dz = x[s] - c.x[i], y[s] - c.y[i], z[s] - c.z[i]
        d = d[i]
        assert np.array_equal(ax[s], ((d[:, 0] + dx * d[:, 3]) + dy * d[:, 6]) + dz * d[:, 7])
        assert np.array_equal(ay[s], ((d[:, 1] + dx * d[:, 6]) + dy * d[:, 4]) + dz * d[:, 8])
        assert np.array_equal(az[s], ((d[:, 2] + dx * d[:, 7]) + dy * d[:, 8]) + dz * d[:, 5])
    finally:
        gp.close()
