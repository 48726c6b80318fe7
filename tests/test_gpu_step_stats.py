"""The counters of mlh_step come back in one copy that runs from the face count over the
padding behind it to the first simulation's time: at every position of the count in
its 256-byte line they are those that the other calls give."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [60, 62, 63, 64, 65, 127, 128, 1000])
@pytest.mark.parametrize("members", [1, 3])
@pytest.mark.parametrize("graph", [False, True])
def test_counters(n, members, graph):
    from meshlesshydro_gb300 import build, ic, runtime
    from meshlesshydro_gb300.config import MFVConfig
    build.build()
    rng = np.random.default_rng(n)

    def one(k):
        p = ic.kelvin_helmholtz(n_side=int(np.ceil(np.sqrt(n / members))) + k, seed=k)
        keep = np.sort(rng.permutation(p.n)[:n // members + (n % members if k == 0 else 0)])
        for name in ("x", "y", "z", "vx", "vy", "vz", "m", "u"):
            setattr(p, name, np.ascontiguousarray(getattr(p, name)[keep]))
        p.kernel_size = 0.33
        return p

    parts = [one(k) for k in range(members)]
    cfg = MFVConfig.kelvin_helmholtz(parts[0])
    s = runtime.Simulation(cfg, parts[0]) if members == 1 else runtime.Simulation(cfg, members=parts)
    assert s.n == n
    s.set_graph_mode(graph)
    t = 0.0
    for steps in (1, 2):
        st = s.step(steps, check=False)
        dt, time = s.member_times()
        assert st.steps == steps and st.dt == dt[0] and st.time == time[0] > t
        t = st.time
        slots = s.get("off")[-1]            # every face has two
        assert 2 * st.faces == st.pair_interactions == slots * steps
        assert st.newton_iterations >= st.faces - np.count_nonzero(s.get("face_iters") <= 0)
    st = s.step(0)
    assert st.steps == 0 and st.dt == s.member_times()[0][0] and st.time == t
    s.close()
