"""A device allocation that fails leaves the context usable: the call returns out-of-memory, and
the next one allocates what is missing and gives the bits of a fresh context.  Every allocation
of the phase is made to fail in turn, on a new context and on one whose buffers have to grow;
with the smaller refinement constant the selection's tables grow within the call as well."""
import numpy as np
import pytest

from apcloud import binding, ics

pytestmark = pytest.mark.gpu

OOM = -3
N, DEPTH = 9000, 12


def _parts(spread):
    """Uniform, or (few cells) all particles at 8 points."""
    rng = np.random.default_rng(5)
    x = rng.random((3, N))
    if not spread:
        x = 0.25 + 0.5 * rng.integers(0, 2, (3, N)) + 1e-9 * x
    z = np.zeros(N)
    return ics.Particles(x[0].copy(), x[1].copy(), x[2].copy(), z.copy(), z.copy(), z.copy())


def _cells(g):
    return [g.codes(), np.array(g.counts())]


def _each_allocation_fails(lib, new, call, got, want, least):
    """new() -> context, call(g) the phase; got(g) must equal want after every failure."""
    for nth in range(1, 1000):
        g = new()
        lib.apc_test_fail_alloc(g.h, nth)
        failed = False
        try:
            call(g)
        except binding.ApcError as e:
            assert e.status == OOM
            failed = True
        lib.apc_test_fail_alloc(g.h, 0)
        call(g)
        assert all(np.array_equal(a, b) for a, b in zip(got(g), want)), nth
        g.close()
        if not failed:
            break
    assert nth > least


@pytest.mark.parametrize("grow", [False, True])
@pytest.mark.parametrize("gfd_c", [2e-3, 5e-5])
def test_select_after_a_failed_allocation(gpu_lib, gfd_c, grow):
    g = binding.GpuPath(_parts(True), DEPTH, gfd_c)
    g.select()
    want = _cells(g)
    g.close()

    def new():
        g = binding.GpuPath(_parts(not grow), DEPTH, gfd_c)
        if grow:
            g.select()
            g.set_particles(_parts(True))
        return g

    lib = binding.load_library(gpu_lib)
    _each_allocation_fails(lib, new, lambda g: g.set_particles(_parts(True)) or g.select(), _cells, want, 10)


@pytest.mark.parametrize("kw", [dict(), dict(restart=200), dict(precision=binding.APC_PREC_MIXED),
                                dict(precision=binding.APC_PREC_MIXED, solve_graphs=0),
                                dict(precision=binding.APC_PREC_MIXED_VCYCLE, mg_reorth=1),
                                dict(precision=binding.APC_PREC_FP64_MULTIGRID)], ids=lambda k: "-".join(map(str, k.values())))
def test_solve_after_a_failed_allocation(gpu_lib, kw):
    n = 6000
    parts = ics.uniform_ball(n, 0.3, seed=3)
    c = 8.0 ** (5.0 / 3.0) * (n / (4.0 / 3.0 * np.pi * 0.3 ** 3)) ** (-2.0 / 3.0)
    few = ics.uniform_ball(n, 0.3, seed=3)  # another state of the box first, whose buffers then grow
    for a in (few.x, few.y, few.z):
        a[:] = 0.5 + 0.2 * (a - 0.5)
    solve = lambda g: g.solve(1.0 / n, 30.0, -1.0)  # noqa: E731
    got = lambda g: [g.fields().density, g.fields().potential, g.fields().deriv]  # noqa: E731

    def new(grow):
        g = binding.GpuPath(few if grow else parts, 21, c, **kw)
        g.select()
        if grow:
            solve(g)
            g.set_particles(parts)
            g.select()
        return g

    g = new(False)
    solve(g)
    want = got(g)
    g.close()
    lib = binding.load_library(gpu_lib)
    _each_allocation_fails(lib, lambda: new(False), solve, got, want, 15)
    _each_allocation_fails(lib, lambda: new(True), solve, got, want, 1)
