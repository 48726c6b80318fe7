"""A tuning without face_split leaves the structure to the size rule, as a context
whose tuning was never set."""
import numpy as np
import pytest

SHAPES = {"face_threads": 128, "face_blocks_per_sm": 8, "grad_threads": 128, "nns_warps_per_sm": 32}


def test_unset_fields():
    from meshlesshydro_gb300 import runtime

    class Lib:
        @staticmethod
        def mlh_set_tuning(handle, t):
            Lib.got = {k: getattr(t._obj, k) for k, _ in runtime.Tuning._fields_}
            return 0

    sim = object.__new__(runtime.Simulation)
    sim.L, sim.h = Lib, None
    sim.set_tuning(SHAPES)
    assert Lib.got == dict(SHAPES, face_split=-1, link_overlap=1, persistent_binning=0, fp32_filters=3, learned_guess=1)


@pytest.mark.gpu
def test_rule_by_size_can_be_set():
    from meshlesshydro_gb300 import build, ic, runtime
    from meshlesshydro_gb300.config import MFVConfig
    build.build()
    p = ic.kelvin_helmholtz(n_side=20, seed=2)
    cfg = MFVConfig.kelvin_helmholtz(p)
    states = []
    for split in (None, -1, 1):
        s = runtime.Simulation(cfg, p)
        if split is not None:
            s.set_tuning(dict(SHAPES, face_split=split))
        for bad in (-2, 3):
            with pytest.raises(runtime.MLHError):
                s.set_tuning(dict(SHAPES, face_split=bad))
        s.step(2)
        states.append(s.get_state())
        s.close()
    for other in states[1:]:
        for k in states[0]:
            np.testing.assert_array_equal(states[0][k], other[k])


# both sides of the rule's line, a million faces: 10 per particle in 2D, 16 in 3D
@pytest.mark.gpu
@pytest.mark.parametrize("dim,n_side", [(2, 323), (2, 324), (3, 40), (3, 41)])
def test_structures_beside_the_line(dim, n_side):
    from meshlesshydro_gb300 import build, ic, runtime
    from meshlesshydro_gb300.config import MFVConfig
    build.build()
    p = ic.kelvin_helmholtz(n_side=n_side, seed=2) if dim == 2 else ic.sedov(n_side=n_side, seed=2)
    cfg = MFVConfig.kelvin_helmholtz(p) if dim == 2 else MFVConfig.sedov(p)
    states = []
    for split in (-1, 0, 2):
        s = runtime.Simulation(cfg, p)
        s.set_tuning(dict(SHAPES, face_split=split))
        s.step(2)
        states.append(s.get_state())
        s.close()
    for other in states[1:]:
        for k in states[0]:
            np.testing.assert_array_equal(states[0][k], other[k])
