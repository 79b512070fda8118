"""The Jacobi-scaled operators of the multigrid paths at stencil sizes that fill the slots of a
thread and that leave a remainder.  Each path solves to the same residual tolerance (1e-10), so the
gradients agree with those of the FP64 path to the 1e-6 RMS that the paths promise."""
import numpy as np
import pytest

from apcloud import binding, ics

PATHS = {"mixed": binding.APC_PREC_MIXED, "vcycle32": binding.APC_PREC_MIXED_VCYCLE,
         "fp64mg": binding.APC_PREC_FP64_MULTIGRID}


@pytest.mark.gpu
@pytest.mark.parametrize("lm", [17, 18, 22, 23, 24])
@pytest.mark.parametrize("path", sorted(PATHS))
def test_scaled_operators_of_every_width(gpu_lib, path, lm):
    cfg = ics.config("ball32k", n=6000, seed=11)
    grads = []
    for prec in (binding.APC_PREC_FP64, PATHS[path]):
        gp = binding.GpuPath(cfg.particles(), cfg.depth, cfg.gfd_c, lm=lm, precision=prec)
        try:
            gp.select()
            gp.solve(1.0, -1.0)
            st = gp.solve_stats()
            assert st["density_reason"] == 2 and st["potential_reason"] == 2
            grads.append(gp.fields().deriv[:, :3])
        finally:
            gp.close()
    a, b = grads
    assert np.sqrt(np.mean((a - b) ** 2)) <= 1e-6 * np.sqrt(np.mean(a ** 2))
