"""A simulation alone and as a member of a large ensemble: the gradients' sums take
another order (8, 4 or 2 lanes per particle alone, one in the ensemble), everything
before them is the same, and the states agree to rounding."""
import numpy as np
import pytest

from helpers import assert_normwise

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side", [23, 90, 140])     # 529, 8100 and 19600 particles: 8, 4 and 2 lanes
def test_member_of_a_large_ensemble(side):
    from meshlesshydro_gb300 import build, ic, runtime
    from meshlesshydro_gb300.config import MFVConfig
    build.build()
    p = ic.kelvin_helmholtz(n_side=side, seed=5)
    others = [ic.kelvin_helmholtz(n_side=120, seed=k) for k in (1, 2)]
    cfg = MFVConfig.kelvin_helmholtz(p)
    alone = runtime.Simulation(cfg, p)
    many = runtime.Simulation(cfg, members=[others[0], p, others[1]])
    assert many.n > 24320
    lo = others[0].n
    alone.step(1)
    many.step(1)
    oa, om = alone.get("off"), many.get("off")
    np.testing.assert_array_equal(oa, om[lo:lo + p.n + 1] - om[lo])
    mask = (1 << 29) - 1
    nm, na = many.get("nnl")[om[lo]:om[lo + p.n]], alone.get("nnl")
    np.testing.assert_array_equal((nm & mask) - lo, na & mask)
    for name in ("rho", "omega", "P"):
        np.testing.assert_array_equal(alone.get(name), many.get(name)[lo:lo + p.n])
    assert alone.member_times()[0][0] == many.member_times()[0][1]
    alone.step(2)
    many.step(2)
    a, b = alone.get_state(), many.get_state()
    for k in a:     # the gate of ensemble members against the oracle after three steps
        assert_normwise(b[k][lo:lo + p.n], a[k], 1e-11, what=k)
    alone.close()
    many.close()
