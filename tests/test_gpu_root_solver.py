"""The Riemann solver's choice by gamma: N-th roots where 2 gamma / (gamma - 1) is
5 or 7 (gamma = 5/3, 7/5), powers for any other gamma, also one next to them.
Fluxes against the oracle's solver, the face-pass structures of the seventh-root
solver bit for bit, and the same step from a gamma that takes the powers."""
from dataclasses import replace

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def faces(rng, n, dim):
    rho, p = 10.0 ** rng.uniform(-3, 3, (2, n, 2))
    v = rng.normal(0.0, 0.5, (n, 2, dim))
    w = [np.concatenate([rho[:, k:k + 1], p[:, k:k + 1], v[:, k]], axis=1) for k in (0, 1)]
    return w[0], w[1], rng.normal(0.0, 0.2, (n, dim)), rng.normal(0.0, 1e-3, (n, dim))


@pytest.mark.parametrize("n", [1, 33, 4097])
@pytest.mark.parametrize("gamma", [7.0 / 5.0, 1.4 + 1e-9, 5.0 / 3.0 - 1e-9, 1.3, 1.5, 2.0])
def test_fluxes_by_gamma(oracle_mod, gamma, n):
    from meshlesshydro_gb300 import build, runtime
    build.build()
    w = faces(np.random.default_rng(7), n, 3)
    Fo, ito, _ = oracle_mod.riemann_fluxes(*w, gamma=gamma)
    Fg, itg, _ = runtime.riemann_fluxes(*w, gamma=gamma)
    ok = ito >= 0
    assert np.array_equal(itg < 0, ~ok) and np.max(np.abs(itg[ok] - ito[ok]), initial=0) <= 1
    # 1e-12 of the largest flux, as for the two gammas of the Riemann tests
    scale = np.maximum(np.max(np.abs(Fo[ok]), axis=0), 1e-300)
    assert np.max(np.abs(Fg[ok] - Fo[ok]) / scale) <= 1e-12


@pytest.mark.parametrize("dim", [2, 3])
def test_seventh_root_structures_and_powers(dim):
    from meshlesshydro_gb300 import build, ic, runtime
    from meshlesshydro_gb300.config import MFVConfig
    build.build()
    if dim == 2:
        p = ic.kelvin_helmholtz(n_side=40, seed=5, gamma=1.4)
        cfg = MFVConfig.kelvin_helmholtz(p)
    else:
        p = ic.sedov(n_side=14, seed=5, gamma=1.4)
        cfg = MFVConfig.sedov(p)

    def state(c, split):
        s = runtime.Simulation(c, p)
        s.set_tuning({"face_threads": 128, "face_blocks_per_sm": 3, "grad_threads": 64, "nns_warps_per_sm": 32,
                      "face_split": split})
        st = s.step(3)
        out = s.get_state()
        s.close()
        return out, st.newton_iterations

    one, it = state(cfg, 0)
    for split in (1, 2):
        other, it2 = state(cfg, split)
        assert it2 == it
        for k in one:
            np.testing.assert_array_equal(one[k], other[k])
    # a gamma of 7/5 (1 + 1e-11) takes the powers: the states differ by the
    # gamma's own change, 1e-11 times a factor of at most 100
    near, _ = state(replace(cfg, gamma=1.4 * (1 + 1e-11)), 0)
    for k in one:
        assert np.max(np.abs(near[k] - one[k])) <= 1e-9 * max(np.max(np.abs(one[k])), 1e-3), k
