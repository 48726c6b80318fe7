"""Results do not depend on the unit of length: a power of two scales every length
exactly, so neighbour lists are the same and densities, smoothing lengths and steps
are the same bits at the other scale, also where the squares of lengths leave the
range of single precision (the search's filter then passes every candidate of the
stencil and the FP64 test decides alone)."""
from dataclasses import replace

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TWO67, TWO40 = 2.0 ** 67, 2.0 ** 40     # 1.5e20, 1.1e12


def scaled(p, s):
    """p with lengths times s; densities, velocities and energies as they are."""
    q = p.copy()
    q.x, q.y, q.z, q.m = q.x * s, q.y * s, q.z * s, q.m * s ** q.dim
    q.kernel_size *= s
    q.box_lo, q.box_hi = tuple(v * s for v in q.box_lo), tuple(v * s for v in q.box_hi)
    return q


def setup(dim, periodic=True):
    from meshlesshydro_gb300 import build, ic
    from meshlesshydro_gb300.config import MFVConfig
    build.build()
    if dim == 2:
        p = ic.kelvin_helmholtz(n_side=23, seed=3)
        return p, lambda q: MFVConfig.kelvin_helmholtz(q, periodic=periodic)
    p = ic.sedov(n_side=16, seed=3, energy=0.05)
    return p, lambda q: MFVConfig.sedov(q, periodic=periodic)


@pytest.mark.parametrize("scale", [TWO67, TWO40, 1 / TWO40, 1 / TWO67])
@pytest.mark.parametrize("periodic", [True, False])
@pytest.mark.parametrize("dim", [2, 3])
def test_lists_and_density(dim, periodic, scale):
    from meshlesshydro_gb300 import runtime
    p, config = setup(dim, periodic)
    got = []
    for q, s in ((p, 1.0), (scaled(p, scale), scale)):
        sim = runtime.Simulation(config(q), q)
        sim.prepare()
        got.append([sim.get("noi"), sim.get("nnl"), sim.get("rho"), sim.get("omega") * s ** dim, sim.get("dt") / s])
        sim.close()
    for a, b in zip(*got):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("scale", [TWO67, 1 / TWO67])
def test_smoothing_lengths(scale):
    from meshlesshydro_gb300 import runtime
    p, config = setup(2)
    got = []
    for q, s in ((p, 1.0), (scaled(p, scale), scale)):
        sim = runtime.Simulation(replace(config(q), adaptive_h=True, n_ngb=14.0), q)
        h, n_eff, clamped = sim.smoothing_lengths(14.0)
        sim.prepare()
        got.append([h / s, n_eff, np.array(clamped), sim.get("noi"), sim.get("nnl"), sim.get("rho")])
        sim.close()
    for a, b in zip(*got):
        np.testing.assert_array_equal(a, b)


# cgs-like units among them: lengths of 1e18, densities of 1e-24, so that gradients of
# the density (1e-41) are below the normal range of single precision.  Powers of 2^10
# keep fifth roots of pressures exact as well.
UNITS = [(2.0 ** 60, 1.0), (2.0 ** 60, 2.0 ** -80), (2.0 ** 60, 2.0 ** -100), (TWO67, 2.0 ** -80), (1 / TWO40, 2.0 ** 40),
         (2.0 ** -60, 1.0), (1 / TWO67, 2.0 ** 80)]


def state_after(cfg, p, steps, s, r, filters):
    from meshlesshydro_gb300 import runtime
    sim = runtime.Simulation(cfg, p)
    sim.set_tuning({"face_threads": 128, "face_blocks_per_sm": 8, "grad_threads": 128, "nns_warps_per_sm": 32,
                    "face_split": 0, "fp32_filters": filters})
    sim.step(steps)
    out = sim.get_state()
    for k in "xyz":
        if k in out:
            out[k] = out[k] / s
    out["m"] = out["m"] / (s ** p.dim * r)
    out["time"] = sim.member_times()[1] / s
    sim.close()
    return out


@pytest.mark.parametrize("s,r", UNITS)
@pytest.mark.parametrize("dim", [2, 3])
def test_steps(dim, s, r):
    p, config = setup(dim)
    rng = np.random.default_rng(8)
    p.u *= rng.uniform(0.5, 2.0, p.n)       # fields without symmetry or flat parts
    p.m *= rng.uniform(0.8, 1.25, p.n)
    q = scaled(p, s)
    q.m = q.m * r
    want = state_after(config(p), p, 3, 1.0, 1.0, 3)
    for filters in (0, 1, 2, 3):
        got = state_after(config(q), q, 3, s, r, filters)
        for k in want:
            np.testing.assert_array_equal(got[k], want[k], err_msg=f"{k}, filters {filters}")


def test_time_step_costs_the_same():
    """The time step's filter works in units of kernelSize: in a large unit of length it
    used to give up, and v_sig of every particle was evaluated in FP64 (the gradients
    and the time step of KH 100^2: 103 us instead of 42)."""
    from meshlesshydro_gb300 import build, ic, runtime
    from meshlesshydro_gb300.config import MFVConfig
    build.build()
    p = ic.kelvin_helmholtz(n_side=100, seed=3)
    ms = []
    for s in (1.0, 2.0 ** 60, 2.0 ** -60):
        q = scaled(p, s)
        sim = runtime.Simulation(MFVConfig.kelvin_helmholtz(q), q)
        sim.step(2)
        sim.set_kernel_timing(True)
        best = np.inf
        for _ in range(5):
            sim.reset_kernel_times()
            sim.step(2)
            best = min(best, sim.kernel_times()["gradients_limiter"][1])
        ms.append(best)
        sim.close()
    assert max(ms) < 1.5 * min(ms), ms
