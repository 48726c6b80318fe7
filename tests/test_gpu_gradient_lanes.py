"""Gradients with several lanes per particle (few particles) against the oracle.

Below about 24 000 particles 2, 4 or 8 lanes of a warp share a particle's
neighbours (Particles::gradient, slopeLimiter, compPsijTilde and
compGlobalTimestep; Particles.cpp:1102-1485).  One step, stage by stage,
at sizes on both sides of each line and at partly filled warps; with lists
beyond the limiter's 64 candidate bits; with the links inside the kernel,
and with the single-precision filters off.
"""
from dataclasses import replace

import pytest

from meshlesshydro_gb300 import ic
from meshlesshydro_gb300.config import MFVConfig
from helpers import compare_step, state_of

pytestmark = pytest.mark.gpu

TUNE = {"face_threads": 128, "face_blocks_per_sm": 8, "grad_threads": 128, "nns_warps_per_sm": 32, "face_split": 0}


# n = 121 ... 24025 and 343 ... 24389: 8 lanes up to 3040, 4 to 10944, 2 to 24320 on 152 SMs
@pytest.mark.parametrize("dim,n_side", [(2, 11), (2, 55), (2, 56), (2, 104), (2, 105), (2, 155), (3, 7), (3, 14),
                                        (3, 15), (3, 22), (3, 23), (3, 28), (3, 29)])
@pytest.mark.parametrize("mode", ["default", "links_inside", "filters_off"])
def test_step_matches_oracle(oracle_mod, dim, n_side, mode):
    _step(oracle_mod, *_setup(dim, n_side), mode)


@pytest.mark.parametrize("mode", ["default", "filters_off"])
@pytest.mark.parametrize("n_side", [12, 16, 22])
def test_long_lists_match_oracle(oracle_mod, n_side, mode):
    p, cfg = _setup(3, n_side)
    _step(oracle_mod, p, replace(cfg, kernel_size=1.45 * cfg.kernel_size, max_neighbours=160), mode)


def _setup(dim, n_side):
    if dim == 2:
        p = ic.kelvin_helmholtz(n_side=n_side, seed=n_side)
        return p, MFVConfig.kelvin_helmholtz(p)
    p = ic.sedov(n_side=n_side, seed=n_side)
    return p, MFVConfig.sedov(p, periodic=True)


def _step(oracle_mod, p, cfg, mode):
    from meshlesshydro_gb300 import build, runtime
    build.build()
    o = oracle_mod.Oracle(cfg, p)
    assert o.step() == 0
    g = runtime.Simulation(cfg, p)
    if mode == "links_inside":
        g.set_tuning(dict(TUNE, link_overlap=2))
    elif mode == "filters_off":
        g.set_tuning(dict(TUNE, fp32_filters=0))
    assert g.step(1).steps == 1
    compare_step(g, o, cfg.dim, slots=True, what=f"{mode}, n = {p.n}: ", pre=state_of(p))
    g.close()
