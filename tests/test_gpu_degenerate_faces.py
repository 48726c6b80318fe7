"""Riemann problems at the edge of what the solver takes: faces without a normal and
NaN velocities.  Sorting the sides of a problem by pressure must not change what is
reported."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

VACUUM = 1 << 6


def problems(n, seed, dim=3):
    rng = np.random.default_rng(seed)
    rho, p = 10.0 ** rng.uniform(-2, 2, (2, 2, n))
    v = rng.normal(0.0, 0.1, (2, n, dim))
    return rho, p, v, rng.normal(0.0, 1e-3, (n, dim)), rng.normal(0.0, 0.2, (n, dim))


def solve(rho, p, v, A, vf, gamma):
    from meshlesshydro_gb300 import build, runtime
    build.build()
    W = [np.concatenate([rho[k][:, None], p[k][:, None], v[k]], axis=1) for k in (0, 1)]
    return runtime.riemann_fluxes(*W, vf, A, gamma=gamma)


# |A|^2 is zero, underflows and overflows: there is no normal, the flux is NaN and
# nothing says vacuum
@pytest.mark.parametrize("scale", [0.0, 1e-160, 1e160])
@pytest.mark.parametrize("gamma", [5.0 / 3.0, 7.0 / 5.0, 1.3])
def test_faces_without_a_normal_are_no_vacuum(gamma, scale):
    rho, p, v, A, vf = problems(64, 3)
    F, it, st = solve(rho, p, v, A * scale, vf, gamma)
    assert st & VACUUM == 0
    assert np.all(np.isnan(F))


@pytest.mark.parametrize("gamma", [5.0 / 3.0, 7.0 / 5.0, 1.3])
def test_nan_velocity_does_not_depend_on_the_sides(gamma):
    rho, p, v, A, vf = problems(64, 4)
    v[0] = np.nan
    F, it, st = solve(rho, p, v, A, vf, gamma)
    up, down = p[0] < p[1], p[0] > p[1]
    assert up.any() and down.any()
    assert len(set(it[up]) | set(it[down])) == 1
