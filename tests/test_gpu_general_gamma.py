"""Whole steps with a gamma that takes the general Riemann solver (powers), stage by
stage against the oracle: gamma = 7/5 and 5/3 take roots, so the set-ups of the other
parity tests do not run these face kernels."""
import pytest

from meshlesshydro_gb300 import ic
from meshlesshydro_gb300.config import MFVConfig
from helpers import compare_step, state_of

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("split", [0, 1, 2])        # structures that only the root solvers have: one pass
@pytest.mark.parametrize("gamma", [1.1, 1.3, 2.0, 3.0])
@pytest.mark.parametrize("name", ["kh", "sedov", "sedov_open", "kh_quadrature"])
def test_step_matches_oracle(oracle_mod, name, gamma, split):
    from meshlesshydro_gb300 import build, runtime
    build.build()
    if name.startswith("kh"):
        p = ic.kelvin_helmholtz(n_side=24, seed=7, gamma=gamma)
        cfg = MFVConfig.kelvin_helmholtz(p, first_order_quad_point=name == "kh")
    else:
        p = ic.sedov(n_side=12, seed=7, energy=0.05, gamma=gamma, periodic=name == "sedov")
        cfg = MFVConfig.sedov(p, periodic=name == "sedov")
    o = oracle_mod.Oracle(cfg, p)
    want = o.step()
    g = runtime.Simulation(cfg, p)
    g.set_tuning({"face_threads": 128, "face_blocks_per_sm": 8, "grad_threads": 128, "nns_warps_per_sm": 32,
                  "face_split": split})
    st = g.step(1, check=False)
    assert st.steps == 1 and (st.status != 0) == (want != 0)
    compare_step(g, o, cfg.dim, slots=True, what=f"{name}, gamma = {gamma}: ", pre=state_of(p))
    g.close()
