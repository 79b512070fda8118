"""apc_set_particles_device / apc_get_particles_device on arrays a kernel uses directly and on
those that take copies (an odd address), in either order with host
uploads: the particles come back as they went in, and a step gives what it gives from host
arrays."""
import ctypes as C

import numpy as np
import pytest

from apcloud import binding, ics

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 255, 4097, 50021])
def test_device_arrays_round_trip(gpu_lib, n):
    import torch

    parts = ics.uniform_ball(n, 0.25, seed=5)
    rng = np.random.default_rng(n)
    host = [a for a in parts.as_tuple()[:3]] + [rng.standard_normal(n) for _ in range(3)]
    c = 8.0 ** (5.0 / 3.0) * (max(n, 64) / (4.0 / 3.0 * np.pi * 0.25 ** 3)) ** (-2.0 / 3.0) if n > 1 else 0.5
    g = binding.GpuPath(parts, 21, c, precision=binding.APC_PREC_MIXED)

    def arrays(odd):
        raw = torch.zeros(6, 8 * n + 64, dtype=torch.uint8, device="cuda")
        off = 4 if odd else 0
        return raw, [raw[k, off:off + 8 * n].data_ptr() for k in range(6)], off

    def read(raw, off):
        return [raw[k, off:off + 8 * n].cpu().numpy().copy().view(np.float64) for k in range(6)]

    def push(raw, off):
        for k in range(6):
            raw[k, off:off + 8 * n] = torch.from_numpy(np.ascontiguousarray(host[k]).view(np.uint8)).cuda()
        torch.cuda.synchronize()

    for odd_in, odd_out in ((False, False), (True, False), (False, True)):
        raw, ptrs, off = arrays(odd_in)
        push(raw, off)
        g.set_particles(ics.Particles(*[h[::-1].copy() for h in host]))  # an upload in flight
        assert g.lib.apc_set_particles_device(g.h, *ptrs) == 0
        out, optrs, ooff = arrays(odd_out)
        assert g.lib.apc_get_particles_device(g.h, *optrs) == 0
        for a, b in zip(read(out, ooff), host):
            assert np.array_equal(a, b)
        if n >= 255:
            want = []
            for how in ("device", "host"):
                if how == "device":
                    assert g.lib.apc_set_particles_device(g.h, *ptrs) == 0
                else:
                    g.set_particles(ics.Particles(*[h.copy() for h in host]))
                g.select()
                g.move_position(0.01, 1.0)
                want.append(g.particles()[:6])
            for a, b in zip(*want):
                assert np.array_equal(a, b)
    # some of the arrays may be left out of a read
    out, optrs, ooff = arrays(False)
    optrs[1] = None
    assert g.lib.apc_get_particles_device(g.h, *[C.c_void_p(p) for p in optrs]) == 0
    g.close()
