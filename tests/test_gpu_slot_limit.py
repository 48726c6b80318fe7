"""The most neighbours a particle can have: the search lists K + 32 candidates per
particle in shared memory, so slots grow to the K that a block can hold (444, and
260 with smoothing lengths, for 227 KB) and a particle with more is refused with
MLH_ERR_CAPACITY before anything reads lists that no search wrote."""
from dataclasses import replace

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

H = 0.3
CAPACITY = 1 << 23


def clump(k, seed):
    """k particles in a ball much smaller than H, 30 spread over the unit cube."""
    from meshlesshydro_gb300 import ic
    rng = np.random.default_rng(seed)
    x = np.concatenate([0.5 + rng.normal(0.0, 0.02, (k, 3)), rng.random((30, 3))])
    n = len(x)
    zero = np.zeros(n)
    return ic.ParticleSet(3, *(np.ascontiguousarray(x[:, a]) for a in range(3)), zero, zero.copy(), zero.copy(),
                          np.full(n, 1.0 / n), np.ones(n), H, (0.0, 0.0, 0.0), (1.0, 1.0, 1.0))


def context(k, adaptive):
    from meshlesshydro_gb300 import build, runtime
    from meshlesshydro_gb300.config import MFVConfig
    build.build()
    p = clump(k, k)
    cfg = MFVConfig.sedov(p)
    if adaptive:
        cfg = replace(cfg, adaptive_h=True, n_ngb=40.0)
    return runtime.Simulation(cfg, p), cfg, p


# 64 slots grow by half: 96, 144, 216, 324 and then 444 (216 and then 260), not 488 (324)
@pytest.mark.parametrize("k,adaptive", [(200, False), (330, False), (420, False), (180, True), (235, True)])
def test_slots_grow_to_the_limit(oracle_mod, k, adaptive):
    from meshlesshydro_gb300 import runtime
    s, cfg, p = context(k, adaptive)
    try:
        s.prepare()
    except runtime.MLHError as e:
        assert e.status == 1 << 8       # one of the 30 has no neighbour, as the oracle says
    o = oracle_mod.Oracle(cfg, p)
    o.step()
    for name in ("off", "noi", "nnl"):
        np.testing.assert_array_equal(s.get(name), o.get(name), err_msg=name)
    s.close()


@pytest.mark.parametrize("k,adaptive", [(500, False), (700, False), (300, True), (500, True)])
def test_more_neighbours_are_refused(k, adaptive):
    from meshlesshydro_gb300 import ic, runtime
    s, cfg, p = context(k, adaptive)
    for call in (s.prepare, lambda: s.step(1), lambda: s.step(2), lambda: s.smoothing_lengths(40.0)):
        with pytest.raises(runtime.MLHError) as e:
            call()
        assert e.value.status & CAPACITY and "slots per particle" in str(e.value)
    # the context serves a state within the limit
    q = p.copy()
    q.x, q.y, q.z = np.random.default_rng(1).random((3, p.n))
    s.set_state(q)
    fresh = runtime.Simulation(cfg, q)
    s.step(1, check=False)
    fresh.step(1, check=False)
    a, b = s.get_state(), fresh.get_state()
    for name in a:
        np.testing.assert_array_equal(a[name], b[name], err_msg=name)
    s.close()
    fresh.close()


@pytest.mark.parametrize("slots", [448, 2000])
def test_configured_slots_above_the_limit_are_refused(slots):
    from meshlesshydro_gb300 import build, ic, runtime
    from meshlesshydro_gb300.config import MFVConfig
    build.build()
    p = ic.sedov(n_side=8, seed=1)
    s = runtime.Simulation(MFVConfig.sedov(p, max_neighbours=slots), p)
    for call in (s.prepare, lambda: s.step(1)):
        with pytest.raises(runtime.MLHError) as e:
            call()
        assert e.value.status & CAPACITY
    assert s.step(0).steps == 0
    s.close()
