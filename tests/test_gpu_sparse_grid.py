"""An open box whose particles spread: most cells of the grid are empty, and the cell
buffers grow under a context that was made for a dense one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def spread(distance, n_side):
    from meshlesshydro_gb300 import ic
    p = ic.sedov(n_side=n_side, seed=3, periodic=False)
    p.x[-2:] += distance        # two that left together
    return p


def context(p):
    from meshlesshydro_gb300 import build, runtime
    from meshlesshydro_gb300.config import MFVConfig
    build.build()
    return runtime.Simulation(MFVConfig.sedov(p, periodic=False), p)


# cells of the grid below, at and above the warps of the sort and the search
@pytest.mark.parametrize("persistent", [0, 1])
@pytest.mark.parametrize("n_side,distance", [(5, 0.0), (9, 20.0), (12, 40.0), (12, 100.0), (12, 1000.0)])
def test_lists(oracle_mod, n_side, distance, persistent):
    from meshlesshydro_gb300.config import MFVConfig
    p = spread(distance, n_side)
    s = context(spread(0.0, n_side))
    s.set_tuning({"face_threads": 128, "face_blocks_per_sm": 8, "grad_threads": 128, "nns_warps_per_sm": 32,
                  "face_split": 0, "persistent_binning": persistent})
    s.step(1, check=False)
    s.set_state(p)              # the buffers grow
    s.step(1, check=False)
    o = oracle_mod.Oracle(MFVConfig.sedov(p, periodic=False), p)
    o.step()
    for name in ("off", "noi", "nnl"):
        np.testing.assert_array_equal(s.get(name), o.get(name), err_msg=name)
    s.close()


def test_search_after_growth_costs_the_same():
    """The parts per cell are chosen by the cells: those of the dense grid made the
    search of the grown one visit every empty cell several times (3.4 million cells:
    830 us instead of 314)."""
    p = spread(1000.0, 33)
    us = []
    for first in (p, spread(0.0, 33)):
        s = context(first)
        s.step(1, check=False)
        s.set_state(p)
        s.step(1, check=False)
        s.set_kernel_timing(True)
        best = np.inf
        for _ in range(4):
            s.reset_kernel_times()
            s.step(1, check=False)
            best = min(best, s.kernel_times()["neighbours_density"][1])
        us.append(best)
        s.close()
    assert us[1] < 1.5 * us[0], us
