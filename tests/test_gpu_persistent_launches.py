"""A solve that does not run on a cluster prepares nothing for one: the persistent solve of a box
and the queued solves of a batch launch as many kernels as on a device without clusters, and
give the same bits."""
import numpy as np
import pytest

from apcloud import binding, ics

pytestmark = pytest.mark.gpu

N = 9000
GFD_C = 8.0 ** (5.0 / 3.0) * (N / (4.0 / 3.0 * np.pi * 0.3 ** 3)) ** (-2.0 / 3.0)
STEP = (0.0075, 1.0 / N, 30.0, -1.0, 1.0, 1.0)


def _parts():
    return ics.uniform_ball(N, 0.3, seed=3)


@pytest.mark.parametrize("precision", [binding.APC_PREC_MIXED, binding.APC_PREC_FP64_MULTIGRID])
@pytest.mark.parametrize("queued", [False, True])
def test_no_cluster_work_beside_persistent_solves(gpu_lib, precision, queued):
    lib, got = binding.load_library(gpu_lib), []
    for off in (0, 1):
        if queued:
            path = binding.BatchPath([(_parts(), dict(depth=21, gfd_c=GFD_C, precision=precision))] * 2,
                                     solve_mode=binding.APC_BATCH_SOLVE_QUEUED)
            boxes = path.boxes
        else:
            path = binding.GpuPath(_parts(), 21, GFD_C, precision=precision, solve_graphs=0)
            boxes = [path]
        for g in boxes:
            lib.apc_test_no_clusters(g.h, off)
        if queued:
            path.step([STEP] * 2)
        else:
            path.step(*STEP)
        got.append([(g.kernel_launches(), [np.array(a) for a in g.particles()]) for g in boxes])
        path.close()
    for (l0, p0), (l1, p1) in zip(*got):
        assert l0 == l1
        assert all(np.array_equal(a, b) for a, b in zip(p0, p1))
