"""Morton keys against the oracle's bisection, bit for bit, over boxes that take the exact scaling
([0, 2^m)) and boxes that take the bisection, with coordinates on, just below and just above
cell boundaries of every level, at and beyond the box's ends, and of tiny size."""
import numpy as np
import pytest

from apcloud import binding, ics

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("depth", [21, 20, 7, 1])
@pytest.mark.parametrize("box", [(0.0, 1.0), (0.0, 4.0), (0.0, 2.0 ** -30), (0.0, 3.0), (-1.0, 1.0), (0.25, 1.25)])
def test_keys_match_bisection(gpu_lib, oracle_lib, box, depth):
    import refbind

    lo, hi = box
    rng = np.random.default_rng(depth)
    w = hi - lo
    g = [lo + w * rng.random(3000)]
    for level in range(1, depth + 1):
        b = lo + w * rng.integers(0, 2 ** level, 40) / 2 ** level
        g += [b, np.nextafter(b, -np.inf), np.nextafter(b, np.inf)]
    g.append(np.array([lo, hi, np.nextafter(hi, lo), np.nextafter(lo, -np.inf), lo - w, hi + w, hi * 3 + 1, 5e-324,
                       -5e-324, -0.0, 1e-300, 1e300, -1e300]))
    a = np.concatenate(g)
    x, y, z = a, rng.permutation(a), rng.permutation(a)
    v = np.zeros(a.size)
    parts = ics.Particles(x.copy(), y.copy(), z.copy(), v, v.copy(), v.copy())
    c = 0.5 * w * w  # the root opens, little else
    gp = binding.GpuPath(parts, depth, c, box=box * 3)
    o = refbind.CpuPath("oracle", parts, depth, c, box=box * 3)
    try:
        assert gp.select() == o.select()
        kg, ig = gp.keys()
        ko, io = o.keys()
        assert np.array_equal(kg, ko)
        back_g, back_o = np.empty_like(kg), np.empty_like(ko)
        back_g[ig], back_o[io] = kg, ko  # each particle's own key
        assert np.array_equal(back_g, back_o)
    finally:
        gp.close()
        o.close()
