"""The autotuner times a launch once: shapes that round to the same grid, block sizes
that a context does not use and structures that its solver does not have are left out,
and what it reports can be set again."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gamma,foqp", [(5.0 / 3.0, True), (5.0 / 3.0, False), (7.0 / 5.0, True), (1.3, True)])
def test_reported_tuning(gamma, foqp):
    from meshlesshydro_gb300 import build, ic, runtime
    from meshlesshydro_gb300.config import MFVConfig
    build.build()
    p = ic.kelvin_helmholtz(n_side=40, seed=3, gamma=gamma)
    cfg = MFVConfig.kelvin_helmholtz(p, first_order_quad_point=foqp)
    a = runtime.Simulation(cfg, p)
    t = a.autotune(1)
    assert t["nns_warps_per_sm"] == 32          # 1600 particles: every grid is the cells' own
    assert t["grad_threads"] == 64              # eight lanes share a particle
    if gamma == 1.3 or not foqp:
        assert t["face_split"] == 0             # the only structure there is
    b = runtime.Simulation(cfg, p)
    b.set_tuning(t)
    a.step(2)
    b.step(2)
    sa, sb = a.get_state(), b.get_state()
    for k in sa:
        np.testing.assert_array_equal(sa[k], sb[k])
    a.close()
    b.close()
