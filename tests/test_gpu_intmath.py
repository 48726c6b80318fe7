"""The integer-pipe products and roots of the kernels (csrc/mlh_intmath.cuh) and
their sums and products as fused multiply-adds: products, sums and square roots
bit for bit the IEEE ones; the fifth and seventh roots within 0.53 ulp (half an
ulp of the last rounding, and a fixed point that carries at least six bits
more, its series cut below 2^-58)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NAMES = ("xmul", "mulr", "addr", "subr", "sqrt", "root5", "rroot5", "root7", "rroot7")


def evaluate(x, y):
    from meshlesshydro_gb300 import build, runtime
    build.build()
    L = runtime.load()
    x, y = np.ascontiguousarray(x), np.ascontiguousarray(y)
    out = np.empty((9, x.size))
    assert L.mlh_probe_int_math(x.size, x.ctypes.data, y.ctypes.data, out.ctypes.data) == 0
    return dict(zip(NAMES, out))


def bits(a):
    return np.where(np.isnan(a), np.nan, a).view(np.uint64)


def operands(kind, rng, n):
    sign = rng.choice([-1.0, 1.0], n)
    if kind == "wide":          # every exponent, past both ends of the product's window
        return sign * np.ldexp(rng.uniform(1, 2, n), rng.integers(-1070, 1023, n))
    if kind == "window":        # the edges of the product's window, 2^-512 and 2^512
        return sign * np.ldexp(1 + rng.integers(0, 8, n) * 2.0 ** -52, rng.choice([-513, -512, -511, 510, 511, 512], n))
    if kind == "powers":        # powers of two and their neighbours: the ends of the roots' estimates
        p = np.ldexp(1.0, rng.integers(-80, 80, n))
        return p * (1 + rng.integers(-4, 5, n) * 2.0 ** -53)
    if kind == "near_one":      # 1 - 2^-k: an estimate on the wrong side of its binade
        return np.ldexp(1 + rng.uniform(-0.5, 0.5, n) * 2.0 ** -rng.integers(0, 52, n), rng.integers(-35, 36, n))
    if kind == "ties":          # short mantissas: exact products and halfway cases
        return sign * np.ldexp(rng.integers(1, 1 << 27, n).astype(float), rng.integers(-30, 30, n))
    return np.resize(np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, 1e-310, 2.2250738585072014e-308,
                               1.7976931348623157e308, 1.0, -1.0, 3.0, 1e-200]), n)


KINDS = ("wide", "window", "powers", "near_one", "ties", "special")


@pytest.mark.parametrize("kind", KINDS)
def test_products_sums_and_square_roots_are_ieee(kind):
    rng = np.random.default_rng(3)
    n = 20000
    x = operands(kind, rng, n)
    y = rng.permutation(operands("special" if kind == "special" else kind, rng, n))
    got = evaluate(x, y)
    with np.errstate(all="ignore"):
        want = {"xmul": x * y, "mulr": x * y, "addr": x + y, "subr": x - y, "sqrt": np.sqrt(x)}
    for k, w in want.items():
        np.testing.assert_array_equal(bits(got[k]), bits(w), err_msg=k)


@pytest.mark.parametrize("kind", KINDS[:5])
def test_roots(kind):
    if np.finfo(np.longdouble).nmant < 63:
        pytest.skip("needs an extended long double for the exact roots")
    rng = np.random.default_rng(4)
    x = np.abs(operands(kind, rng, 20000))
    x = x[x >= 2.2250738585072014e-308]
    got = evaluate(x, np.ones_like(x))
    lx = x.astype(np.longdouble)
    for k, num, den in (("root5", 1, 5), ("rroot5", -1, 5), ("root7", 1, 7), ("rroot7", -1, 7)):
        e = lx ** (np.longdouble(num) / den)
        # one Newton step, so that the long double pow need not be trusted to its last bits
        e = e - (e ** (den * num) - lx) / (np.longdouble(den * num) * e ** (den * num - 1))
        err = np.abs(got[k].astype(np.longdouble) - e) / np.spacing(e.astype(np.float64))
        assert float(err.max()) <= 0.53, (k, float(err.max()), x[np.argmax(err)])


def test_roots_of_special_values():
    x = np.array([0.0, np.inf, np.nan, 5e-324, 1e-310])
    got = evaluate(x, x)
    for k, a in (("root5", 0.2), ("rroot5", -0.2), ("root7", 1 / 7), ("rroot7", -1 / 7)):
        with np.errstate(all="ignore"):
            np.testing.assert_allclose(got[k], x ** a, rtol=1e-13, err_msg=k)
