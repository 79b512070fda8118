"""The FP64 GMRES on clusters is the persistent kernel's solve bit for bit, for every cluster size
and both places of the basis, and its cluster size is part of the kernel: a launch cannot lose
it (a profiler that replays cooperative launches drops the launch's cluster attribute, and the
solve then ended at max_it with a wrong density)."""
import numpy as np
import pytest

from apcloud import binding, ics

pytestmark = pytest.mark.gpu

FORMS = [16, 8, 4, -16, -8, -4, -2]


@pytest.mark.parametrize("form", FORMS)
def test_cluster_size_is_compiled_in(gpu_lib, form):
    assert binding.load_library(gpu_lib).apc_test_gmres_cluster_width(0, form) == abs(form)


@pytest.mark.parametrize("restart", [5, 30, 31, 32, 200, 255])
@pytest.mark.parametrize("n", [300, 900, 4096, 20011])
def test_forms_agree_bit_for_bit(gpu_lib, n, restart):
    parts = ics.uniform_ball(n, 0.25, seed=1)
    gfd_c = 8.0 ** (5.0 / 3.0) * (n / (4.0 / 3.0 * np.pi * 0.25 ** 3)) ** (-2.0 / 3.0)
    lib = binding.load_library(gpu_lib)
    ref, ran = None, set()
    for form in [1, 0] + FORMS:
        g = binding.GpuPath(parts, 21, gfd_c, restart=restart, max_it=600)
        try:
            lib.apc_test_gmres_form(g.h, form)
            g.select()
            g.solve(1.0 / n, 30.0)
            if lib.apc_test_gmres_form(g.h, form):
                ran.add(form)
            st, f = g.solve_stats(), g.fields()
        finally:
            g.close()
        got = {k: st[k] for k in st if k.endswith(("its", "reason", "rnorm"))}
        if ref is None:
            ref = (got, f)
            continue
        assert got == ref[0], form
        assert np.array_equal(f.density, ref[1].density) and np.array_equal(f.potential, ref[1].potential), form
    assert 0 in ran and 1 not in ran
    assert len(ran) >= 2  # a form on clusters was set against the persistent kernel
