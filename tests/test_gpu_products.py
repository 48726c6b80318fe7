"""Integer-pipe products at the edges of their window (exponents 2^-256 .. 2^256, beyond
which they are left to the FP64 pipe): the IEEE products bit for bit on both sides of
each edge and for every pairing of an inner with an outer factor."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_products_at_the_window():
    from meshlesshydro_gb300 import build, runtime
    build.build()
    L = runtime.load()
    rng = np.random.default_rng(21)
    m = np.array([1.0, 1 + 2.0 ** -52, 1 + 2.0 ** -26, 1.5, 2 - 2.0 ** -26, 2 - 2.0 ** -52])
    e = np.array([-258, -257, -256, -255, -1, 0, 1, 254, 255, 256, 257])
    one = np.ldexp(m[:, None], e[None, :]).ravel()
    one = np.concatenate([one, -one])
    x, y = (a.ravel() for a in np.meshgrid(one, one))
    # random mantissas at the same exponents
    k = 40000
    x = np.concatenate([x, np.ldexp(rng.uniform(1, 2, k), rng.choice(e, k))])
    y = np.concatenate([y, np.ldexp(rng.uniform(1, 2, k), rng.choice(e, k))])
    out = np.empty((9, x.size))
    assert L.mlh_probe_int_math(x.size, x.ctypes.data, y.ctypes.data, out.ctypes.data) == 0
    np.testing.assert_array_equal(out[0].view(np.uint64), (x * y).view(np.uint64))
    np.testing.assert_array_equal(out[1].view(np.uint64), (x * y).view(np.uint64))
