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
