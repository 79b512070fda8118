"""The work that users of the gravity step have it do, as cases to be timed.

A case is a dict of plain values.  Its "op" is the call sequence:

  step    one Controller step on device arrays: apc_set_particles_device, apc_step,
          apc_get_particles_device.  The whole path: octree, selection, GFD assembly, both
          solves, differentiation, interpolation, kick, drift.
  host    the same through host buffers (pinned), the way the C++ drop-in and the VTK
          tools hold their particles: set_particles, step, get_particles.
  start   Controller.start: select, then the initial half drift (no solve).
  batch   one step of many uneven boxes together (apc_batch_step).
  vjp     forward trajectory and vector-Jacobian product with checkpoints
          (apc_trajectory_vjp): the gradient of a loss on the final state.
  kick    interpolation + kick on caller-owned buffers (apc_move_velocity_noalloc).

Particle sets are the repository's two kinds: cold uniform balls, and Zel'dovich lattices
(a Gaussian random field with a power-law spectrum).  Larger rms displacements stand for
later times: past shell crossing the octree is deep and its cells uneven.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ap-cloud-cosmology_b200"))

from apcloud import binding, ics  # noqa: E402

PRECISION = {"fp64": binding.APC_PREC_FP64, "mixed": binding.APC_PREC_MIXED,
             "fp64mg": binding.APC_PREC_FP64_MULTIGRID, "vcycle32": binding.APC_PREC_MIXED_VCYCLE}
# tree depth (key levels), stencil size and background of every workload here
DEPTH, LM = 21, 17


# ------------------------------------------------------------------------ cases

def listed():
    return [
        # the smallest box of a batch on its own: a step that is launches and round trips
        dict(name="step-ball-4k-mixed", op="step", kind="ball", n=4096, radius=0.3, precision="mixed", a=0.05,
             omega0=1.0, restart=30),
        # the cold collapse of the plain FP64 method, the library's default precision
        dict(name="step-ball-32k-fp64", op="step", kind="ball", n=32768, radius=0.25, precision="fp64", a=0.11,
             omega0=1.0, restart=30),
        # the FP64 method with the restart of the reference's production runs, an odd lattice
        dict(name="step-zel-23-fp64-r200", op="step", kind="zel", side=23, rms=0.25, index=-2.0, precision="fp64",
             a=0.05, omega0=1.0, restart=200),
        # a box of ordinary size on the fastest solver path
        dict(name="step-zel-48-vcycle32", op="step", kind="zel", side=48, rms=0.3, index=-2.0, precision="vcycle32",
             a=0.05, omega0=1.0, restart=30),
        # the Einstein-de Sitter box with host-resident particles, on the mixed path
        dict(name="host-zel-64-mixed", op="host", kind="zel", side=64, rms=0.5, index=-2.0, precision="mixed", a=0.05,
             omega0=1.0, restart=30),
        # a compact ball: more cells than particles (vacuum cells around it), many levels
        dict(name="step-ball-262k-fp64mg", op="step", kind="ball", n=262144, radius=0.18, precision="fp64mg", a=0.05,
             omega0=1.0, restart=30),
        # the headline LambdaCDM box at its first steps
        dict(name="step-zel-128-vcycle32", op="step", kind="zel", side=128, rms=0.7, index=-1.5,
             precision="vcycle32", a=0.047, omega0=0.3, restart=30),
        # the same box at a late time: collapsed regions, a deep tree with uneven cells
        dict(name="step-zel-128-late", op="step", kind="zel", side=128, rms=2.5, index=-1.5, precision="vcycle32",
             a=0.5, omega0=0.3, restart=30),
        # the first calls of a run: octree and selection of two million particles, half drift
        dict(name="start-zel-128", op="start", kind="zel", side=128, rms=0.3, index=-1.5, precision="vcycle32",
             a=0.02, omega0=0.3, restart=30),
        # independent realisations of uneven size stepped together
        dict(name="batch-16-mixed", op="batch", boxes=16, sides="16,24,32,48", pick=2024, precision="mixed", a=0.05),
        # the gradient of a loss on final positions through a short trajectory
        dict(name="vjp-zel-32-8-steps", op="vjp", kind="zel", side=32, rms=0.2, index=-2.0, precision="mixed", a=0.05,
             omega0=1.0, steps=8, every=4),
        # an embedder's interpolation + kick on its own buffers
        dict(name="kick-1m", op="kick", n=1000003, per_cell=9),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges: sizes spread over their logarithm, odd ones among
    them (a ball takes any particle count, a lattice any side)."""
    op = rng.choice(["step", "step", "step", "step", "host", "start", "batch", "vjp", "kick"])
    if op == "kick":
        return dict(op=op, n=_log_int(rng, 3000, 1 << 20), per_cell=rng.randint(3, 40))
    if op == "batch":
        return dict(op=op, boxes=rng.randint(3, 16), sides="16,24,32", pick=rng.randint(1, 10 ** 6),
                    precision=rng.choice(["mixed", "vcycle32"]), a=round(rng.uniform(0.05, 0.4), 3))
    if op == "vjp":
        steps = rng.randint(2, 6)
        return dict(op=op, kind="zel", side=_log_int(rng, 12, 32), rms=round(rng.uniform(0.1, 0.4), 3), index=-2.0,
                    precision="mixed", a=0.05, omega0=1.0, steps=steps, every=rng.randint(1, steps))
    precision = rng.choice(["fp64", "mixed", "fp64mg", "vcycle32", "vcycle32"])
    case = dict(op=op, precision=precision, a=round(rng.uniform(0.04, 0.8), 3), omega0=rng.choice([1.0, 0.3]),
                restart=30)
    if precision == "fp64":
        case["restart"] = rng.choice([30, 30, 200])
    if rng.random() < 0.4:
        case.update(kind="ball", n=_log_int(rng, 2000, 30000 if precision == "fp64" else 250000),
                    radius=round(rng.uniform(0.15, 0.35), 3))
    else:
        # the FP64 method without multigrid does not converge on the large lattices
        side = _log_int(rng, 12, 28 if precision == "fp64" and op != "start" else 110)
        case.update(kind="zel", side=side, rms=round(rng.uniform(0.1, 2.0), 3), index=rng.choice([-2.0, -1.5]))
    return case


# ---------------------------------------------------------------------- inputs

def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _ball(n, radius, g):
    """n points uniform in a sphere at rest; (6, n)."""
    d = torch.randn(3, n, dtype=torch.float64, device="cuda", generator=g)
    d = d / d.norm(dim=0, keepdim=True)
    r = radius * torch.rand(n, dtype=torch.float64, device="cuda", generator=g) ** (1.0 / 3.0)
    return torch.cat([0.5 + d * r, torch.zeros(3, n, dtype=torch.float64, device="cuda")])


def _zeldovich(side, index, rms_spacing, a, omega0, g):
    """Lattice + Zel'dovich displacement of the given rms (in spacings) with growing-mode
    momenta, as ics.zeldovich makes them, on the GPU; (6, side^3)."""
    n = side
    kw = dict(dtype=torch.float64, device="cuda")
    wk = torch.fft.rfftn(torch.randn(n, n, n, generator=g, **kw))
    kx = 2.0 * math.pi * torch.fft.fftfreq(n, d=1.0 / n, **kw)
    kz = 2.0 * math.pi * torch.fft.rfftfreq(n, d=1.0 / n, **kw)
    k3 = torch.meshgrid(kx, kx, kz, indexing="ij")
    k2 = k3[0] ** 2 + k3[1] ** 2 + k3[2] ** 2
    k2[0, 0, 0] = 1.0
    k = k2.sqrt()
    dk = wk * (k ** (0.5 * index) * torch.exp(-0.5 * (k / (0.5 * math.pi * n)) ** 2)) / k2
    dk[0, 0, 0] = 0.0
    psi = torch.stack([torch.fft.irfftn(1j * q * dk, s=(n, n, n)) for q in k3])
    psi = psi * (rms_spacing / n / (psi ** 2).sum(0).mean().sqrt())
    q = (torch.arange(n, **kw) + 0.5) / n
    pos = torch.stack(torch.meshgrid(q, q, q, indexing="ij")) + psi
    pos = pos - torch.floor(pos)
    pos = torch.where(pos >= 1.0, pos - 1.0, pos)
    d, dd = ics.growth(a, omega0, 1.0 - omega0)
    fac = a * a * (dd / d) / ics.kick_factor(a, omega0, 1.0 - omega0)
    return torch.cat([pos.reshape(3, -1), (fac * psi).reshape(3, -1)]).contiguous()


def _particles(case, seed):
    g = _generator(seed)
    if case["kind"] == "ball":
        return _ball(case["n"], case["radius"], g)
    return _zeldovich(case["side"], case["index"], case["rms"], case["a"], case["omega0"], g)


def _gfd_c(case, n):
    """The refinement constant for 8 particles per cell, 16 in the largest lattices."""
    if case["kind"] == "ball":
        rho = n / (4.0 / 3.0 * math.pi * case["radius"] ** 3)
        return 8.0 ** (5.0 / 3.0) * rho ** (-2.0 / 3.0)
    if n >= 100 ** 3:
        return 16.0 ** (5.0 / 3.0) * n ** (-2.0 / 3.0)
    return 1.28 * 8.0 ** (5.0 / 3.0) * n ** (-2.0 / 3.0)


def _constants(n, a, dt, omega0):
    """(dt, c_dens, c_pot, c_field, c_vel, c_pos) of one step at expansion factor a."""
    omegal = 1.0 - omega0
    return (dt, 1.0 / n, 1.5 * omega0 / a, -1.0, ics.kick_factor(a, omega0, omegal),
            ics.drift_factor(a + dt / 2, omega0, omegal))


class _Empty:
    """The argument of GpuPath that names the particle count and holds first particles."""

    def __init__(self, state):
        self.n = int(state.shape[1])
        self._arrays = tuple(state.cpu().numpy())

    def as_tuple(self):
        return self._arrays


def _ptrs(t):
    return [t[k].data_ptr() for k in range(t.shape[0])]


def _context(case, state):
    n = int(state.shape[1])
    return binding.GpuPath(_Empty(state), DEPTH, _gfd_c(case, n), LM, precision=PRECISION[case["precision"]],
                           restart=case.get("restart", 30))


DT = 0.0075  # a step of the named runs is 0.0077 to 0.015 in expansion factor


def prepare(case, seed):
    op = case["op"]
    if op == "kick":
        return _prepare_kick(case, seed)
    if op == "batch":
        return _prepare_batch(case, seed)
    state = _particles(case, seed)
    n = int(state.shape[1])
    st = dict(op=op, path=_context(case, state), state=state, n=n, out=torch.empty_like(state))
    if op == "vjp":
        gen = _generator(seed + 1)
        # the cotangent of a mean squared distance to a perturbed target
        cot = torch.zeros_like(state)
        cot[:3] = 2.0 / n * 0.01 / case["side"] * torch.randn(3, n, dtype=torch.float64, device="cuda", generator=gen)
        a, steps = case["a"], []
        for k in range(case["steps"]):
            steps.append(_constants(n, a + DT * (k + 0.5), DT, case["omega0"]))
        st.update(steps=steps, start=(0.5 * DT, ics.drift_factor(a, case["omega0"], 1.0 - case["omega0"])),
                  every=case["every"], cot0=cot, cot=torch.empty_like(cot))
    elif op == "start":
        st["half"] = (0.5 * DT, ics.drift_factor(case["a"], case["omega0"], 1.0 - case["omega0"]))
    else:
        st["params"] = _constants(n, case["a"], DT, case["omega0"])
        if op == "host":
            st["in"] = state.cpu().pin_memory()
            st["host_out"] = torch.empty((9, n), dtype=torch.float64).pin_memory()
    return st


def _prepare_batch(case, seed):
    rng = np.random.default_rng(case["pick"])
    sides = [int(v) for v in case["sides"].split(",")]
    boxes, states, params = [], [], []
    for b in range(case["boxes"]):
        side = int(rng.choice(sides))
        sub = dict(kind="zel", side=side, rms=float(rng.uniform(0.1, 0.3)), index=-2.0, a=case["a"], omega0=1.0)
        if b % 2 == 0:
            sub = dict(kind="ball", n=side ** 3, radius=float(rng.uniform(0.15, 0.35)), a=case["a"], omega0=1.0)
        s = _particles(sub, seed * 1000 + b)
        n = int(s.shape[1])
        boxes.append((_Empty(s), dict(depth=DEPTH, gfd_c=_gfd_c(sub, n), lm=LM, precision=PRECISION[case["precision"]])))
        states.append(s)
        params.append(_constants(n, case["a"], DT, 1.0))
    # one output array, a slice of columns for each box
    total = sum(int(s.shape[1]) for s in states)
    out = torch.empty((6, total), dtype=torch.float64, device="cuda")
    outs, at = [], 0
    for s in states:
        outs.append(out[:, at:at + s.shape[1]])
        at += int(s.shape[1])
    return dict(op="batch", path=binding.BatchPath(boxes), states=states, params=params, out=out, outs=outs)


def _prepare_kick(case, seed):
    """Particles in cell order, cells of uneven counts (some empty), and the cells' fields,
    as a select and a solve leave them."""
    g = _generator(seed)
    n = case["n"]
    m = max(1, n // case["per_cell"])
    kw = dict(dtype=torch.float64, device="cuda", generator=g)
    cell = torch.sort(torch.randint(0, m, (n,), device="cuda", generator=g))[0]
    count = torch.bincount(cell, minlength=m)
    first = torch.cumsum(count, 0) - count
    centre = torch.rand(3, m, **kw)
    h = 1.0 / round(m ** (1.0 / 3.0) + 1)
    x = centre[:, cell] + h * (torch.rand(3, n, **kw) - 0.5)
    return dict(op="kick", lib=binding.load_library(), n=n, m=m, first=first.int(), count=count.int(), centre=centre,
                deriv=torch.randn(m, 9, **kw), x=x.contiguous(), v0=0.1 * torch.randn(3, n, **kw), cell=cell,
                v=torch.empty(3, n, dtype=torch.float64, device="cuda"),
                acc=torch.empty(3, n, dtype=torch.float64, device="cuda"))


# ------------------------------------------------------------------------ run

def run(state):
    op = state["op"]
    if op == "kick":
        return _run_kick(state)
    if op == "batch":
        return _run_batch(state)
    g = state["path"]
    if op == "host":
        g._check(g.lib.apc_set_particles(g.h, *_ptrs(state["in"])), "apc_set_particles")
        cells, dv, dx = g.step(*state["params"])
        g._check(g.lib.apc_get_particles(g.h, *_ptrs(state["host_out"])), "apc_get_particles")
        return dict(cells=cells, dv=dv, dx=dx, particles=state["host_out"])
    if op == "vjp":
        state["cot"].copy_(state["cot0"])
        torch.cuda.current_stream().synchronize()  # the library reads it on streams of its own
        g.trajectory_vjp(state["steps"], *state["start"], state["every"], _ptrs(state["state"]), _ptrs(state["cot"]),
                         _ptrs(state["out"]))
        return dict(grad=state["cot"], particles=state["out"])
    g._check(g.lib.apc_set_particles_device(g.h, *_ptrs(state["state"])), "apc_set_particles_device")
    if op == "start":
        cells = g.select()
        dx = g.move_position(*state["half"])
        got = dict(cells=cells, dx=dx)
    else:
        cells, dv, dx = g.step(*state["params"])
        got = dict(cells=cells, dv=dv, dx=dx)
    g._check(g.lib.apc_get_particles_device(g.h, *_ptrs(state["out"])), "apc_get_particles_device")
    got["particles"] = state["out"]
    return got


def _run_batch(state):
    path = state["path"]
    for g, s in zip(path.boxes, state["states"]):
        g._check(g.lib.apc_set_particles_device(g.h, *_ptrs(s)), "apc_set_particles_device")
    dv, dx = path.step(state["params"])
    for g, o in zip(path.boxes, state["outs"]):
        g._check(g.lib.apc_get_particles_device(g.h, *_ptrs(o)), "apc_get_particles_device")
    return dict(dv=dv, dx=dx, particles=state["out"])


KICK = (DT, 1.7)  # dt, c_vel


def _run_kick(state):
    import ctypes

    state["v"].copy_(state["v0"])
    dv = ctypes.c_double()
    rc = state["lib"].apc_move_velocity_noalloc(
        state["n"], state["m"], state["first"].data_ptr(), state["count"].data_ptr(), *_ptrs(state["centre"]),
        state["deriv"].data_ptr(), *_ptrs(state["x"]), *_ptrs(state["v"]), *_ptrs(state["acc"]), *KICK,
        ctypes.byref(dv), torch.cuda.current_stream().cuda_stream)
    if rc != 0:
        raise RuntimeError("apc_move_velocity_noalloc: %d" % rc)
    return dict(dv=dv.value, v=state["v"], acc=state["acc"])


# ----------------------------------------------------------------- work, exact

def _count(case):
    return case["n"] if "n" in case else case["side"] ** 3


def work(case):
    op = case["op"]
    if op == "kick":
        m = max(1, case["n"] // case["per_cell"])
        return dict(bytes=case["n"] * (24 + 48 + 24) + m * (8 + 24 + 72), flops=case["n"] * 35.0)
    if op == "batch":
        rng = np.random.default_rng(case["pick"])
        sides = [int(v) for v in case["sides"].split(",")]
        n = 0
        for b in range(case["boxes"]):
            n += int(rng.choice(sides)) ** 3
            rng.uniform()
        steps = 1
    else:
        n, steps = _count(case), case.get("steps", 1)
    if op == "start":
        return dict(bytes=n * 96.0, flops=n * 10.0)
    # per step the particles in and out; per cell (about one for eight particles) a least-squares
    # fit of 17 rows in 9 unknowns and its application
    per = 96.0 + (24.0 if op == "host" else 0.0)
    if op == "vjp":
        return dict(bytes=n * 4 * 48.0, flops=steps * (n * 100.0 + n / 8 * 6000.0))
    return dict(bytes=n * per, flops=steps * (n * 50.0 + n / 8 * 6000.0))


def exact(case, seed):
    """In 64 bits with torch: the half drift of "start" and the whole of "kick".  A step's
    outputs come from the selected octree cells, their ordered stencils and two linear
    solves; rebuilding those cell by cell in plain Python takes minutes, so they have none."""
    if case["op"] == "start":
        s = _particles(case, seed)
        dt, c_pos = 0.5 * DT, ics.drift_factor(case["a"], case["omega0"], 1.0 - case["omega0"])
        x = s[:3] + s[3:] * c_pos * dt
        x = torch.where(x >= 1.0, x - 1.0, x)
        x = torch.where(x < 0.0, x + 1.0, x)
        dx = math.sqrt(float((s[3:] ** 2).sum(0).max())) * c_pos * dt
        return dict(cells=None, dx=dx, particles=torch.cat([x, s[3:]]))
    if case["op"] == "kick":
        p = _prepare_kick(case, seed)
        d, c = p["deriv"], p["cell"]
        dx, dy, dz = p["x"] - p["centre"][:, c]
        d = d[c]
        acc = torch.stack([d[:, 0] + dx * d[:, 3] + dy * d[:, 6] + dz * d[:, 7],
                           d[:, 1] + dx * d[:, 6] + dy * d[:, 4] + dz * d[:, 8],
                           d[:, 2] + dx * d[:, 7] + dy * d[:, 8] + dz * d[:, 5]])
        dv = math.sqrt(float((acc ** 2).sum(0).max())) * KICK[0] * KICK[1]
        return dict(dv=dv, v=p["v0"] + acc * KICK[1] * KICK[0], acc=acc)
    return None
