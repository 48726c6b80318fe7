"""The neighbour search's units: cells split over several warps (few cells), cells
with more particles than a batch, candidate sequences past the registers' 128,
rows that overflow and grow, images at the end of a full row.  Random particles
(uneven cells), lists bit for bit those of the oracle, densities to 1e-12."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def random_set(dim, n, h, seed, clump):
    from meshlesshydro_gb300 import ic
    rng = np.random.default_rng(seed)
    x = rng.random((n, dim))
    if clump:       # up to 230 particles (what the search's shared memory can list) in a ball of one
                    # cell's size, across a corner of the box
        k = min(n // 3, 230)
        x[:k] = np.mod(rng.normal(0.0, 0.25 * h, (k, dim)), 1.0)
    z = np.zeros(n)
    col = [np.ascontiguousarray(x[:, a]) if a < dim else z.copy() for a in range(3)]
    v = [rng.normal(0.0, 0.1, n) if a < dim else z.copy() for a in range(3)]
    return ic.ParticleSet(dim, *col, *v, np.full(n, 1.0 / n), rng.uniform(1.0, 2.0, n), h,
                          (0.0, 0.0, 0.0), (1.0, 1.0, 1.0 if dim == 3 else 0.0))


# 24 slots: the clumps (about 250 neighbours) need six of the eight growths by half
@pytest.mark.parametrize("slots", [0, 24])
@pytest.mark.parametrize("clump", [False, True])
@pytest.mark.parametrize("periodic", [True, False])
@pytest.mark.parametrize("dim,n,h", [(2, 60, 0.33), (2, 700, 0.12), (2, 3000, 0.05), (3, 90, 0.33), (3, 2000, 0.19),
                                     (3, 6000, 0.1)])
def test_lists_and_density(oracle_mod, dim, n, h, periodic, clump, slots):
    from meshlesshydro_gb300 import build, runtime
    from meshlesshydro_gb300.config import MFVConfig
    build.build()
    p = random_set(dim, n, h, 100 * n + dim, clump)
    make = MFVConfig.kelvin_helmholtz if dim == 2 else MFVConfig.sedov
    cfg = make(p, max_neighbours=slots) if dim == 3 else make(p, max_neighbours=slots, periodic=periodic)
    if dim == 3:
        from dataclasses import replace
        cfg = replace(cfg, periodic=periodic)
    o = oracle_mod.Oracle(cfg, p)
    o.step()
    s = runtime.Simulation(cfg, p)
    try:
        s.prepare()
    except runtime.MLHError:
        pass        # particles without neighbours, as the oracle's status says
    for k in ("off", "noi", "nnl"):
        np.testing.assert_array_equal(s.get(k), o.get(k), err_msg=k)
    for k in ("omega", "rho"):     # the per-element gate of the parity tests
        assert np.all(np.abs(s.get(k) - o.get(k)) <= 1e-12 * np.abs(o.get(k))), k
    s.close()
