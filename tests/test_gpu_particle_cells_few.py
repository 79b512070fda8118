"""The particle -> cell map of the kick with every number of cells per warp (32 down to 1, by the
mean count) and uneven cells: given the fields, the accelerations are the interpolation's own
operations, so the comparison is bit for bit."""
import numpy as np
import pytest

from apcloud import binding, ics


@pytest.mark.gpu
@pytest.mark.parametrize("n", [512 * 8, 512 * 8 + 1, 512 * 32 + 1, 512 * 64, 512 * 64 + 1, 512 * 128 + 1, 512 * 300, 512 * 1100])
def test_kick_takes_each_particle_from_its_cell(gpu_lib, n):
    rng = np.random.default_rng(n)
    x = rng.random((3, n))
    x[:, : n // 8] *= 0.5  # uneven cells
    z = np.zeros(n)
    p = ics.Particles(x[0].copy(), x[1].copy(), x[2].copy(), z, z.copy(), z.copy())
    gp = binding.GpuPath(p, 3, 1e-3, precision=binding.APC_PREC_MIXED)  # 512 cells
    try:
        gp.select()
        gp.solve(1.0, -1.0)
        gp.move_velocity(0.01, 1.0)
        c, d = gp.cells(), gp.fields().deriv
        assert c.m == 512
        order = gp.keys()[1]  # the cells' ranges count particles in key order
        x, y, z, _, _, _, ax, ay, az = (q[order] for q in gp.particles())
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
