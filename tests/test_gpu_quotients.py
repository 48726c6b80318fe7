"""The kernels' correctly rounded reciprocal and quotient (mlh_intmath.cuh) against the
IEEE ones, and the reciprocal and reciprocal square root that carry 0.52 ulp, at the
operands where they are most likely wrong: quotients next to a rounding midpoint,
divisors whose reciprocal lies next to one, powers of two and their neighbours, the
edges of the window 2^-256 .. 2^256, and everything that leaves the straight path."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def evaluate(a, b):
    from meshlesshydro_gb300 import build, runtime
    build.build()
    L = runtime.load()
    a, b = np.ascontiguousarray(a, dtype=np.float64), np.ascontiguousarray(b, dtype=np.float64)
    out = np.empty((4, a.size))
    assert L.mlh_probe_quotients(a.size, a.ctypes.data, b.ctypes.data, out.ctypes.data) == 0
    return dict(zip(("rcp_rn", "div_rn", "rcp", "rsqrt"), out))


def bits(x):
    return np.where(np.isnan(x), np.nan, x).view(np.uint64)


def nearest_midpoints(divisors, offsets):
    """(A, B) of 53 bits with A 2^s / B = M + k / B, M odd and of 54 bits: quotients whose
    distance from the midpoint M of two doubles is k of the smallest there is."""
    out = []
    for B in divisors:
        inv = pow(B, -1, 1 << 54)
        for k in offsets:
            for s in (53, 54):
                M = (-k * inv) % (1 << s) | (1 << 53)     # M B = -k mod 2^s, top bit set
                if M % 2 == 0 or (M * B + k) % (1 << s):
                    continue
                A = (M * B + k) >> s
                if 1 << 52 <= A < 1 << 53:
                    out.append((A, B))
    return out


@pytest.mark.parametrize("kind", ["just below two", "random", "all"])
def test_quotients_next_to_midpoints(kind):
    rng = np.random.default_rng(11)
    if kind == "just below two":        # the reciprocal of 2 - j 2^-52 is next to a midpoint itself
        B = [(1 << 53) - j for j in range(1, 6000, 2)] + [(1 << 53) - 2 * int(j) - 1 for j in rng.integers(1, 1 << 23, 3000)]
    elif kind == "random":
        B = [int(b) | 1 for b in rng.integers(1 << 52, 1 << 53, 6000)]
    else:
        B = [(1 << 52) + 2 * j + 1 for j in range(2000)] + [3 << 51 | 1, (3 << 51) - 1, 5 << 50 | 1]
    pairs = nearest_midpoints(B, (1, -1, 3, -3))
    assert len(pairs) > 4000
    a = np.array([float(A) for A, _ in pairs]) * np.ldexp(1.0, rng.integers(-250, 200, len(pairs)) - 52)
    b = np.array([float(B) for _, B in pairs]) * np.ldexp(1.0, rng.integers(-250, 200, len(pairs)) - 52)
    sign = rng.choice([-1.0, 1.0], len(pairs))
    got = evaluate(a * sign, b)
    np.testing.assert_array_equal(bits(got["div_rn"]), bits(a * sign / b))
    np.testing.assert_array_equal(bits(got["rcp_rn"]), bits(1.0 / b))


def operands(kind, rng, n):
    sign = rng.choice([-1.0, 1.0], n)
    if kind == "wide":
        return sign * np.ldexp(rng.uniform(1, 2, n), rng.integers(-1074, 1024, n))
    if kind == "window":        # both ends of the window's binades, from either side
        m = rng.choice([1.0, 1 + 2.0 ** -52, 1.5, 2 - 2.0 ** -52], n)
        return sign * np.ldexp(m, rng.choice([-258, -257, -256, -255, 254, 255, 256, 257], n))
    if kind == "powers":
        return sign * np.ldexp(1 + rng.integers(-4, 5, n) * 2.0 ** -53, rng.integers(-240, 240, n))
    if kind == "reciprocal ends":   # exponents where 1/b leaves the normal numbers
        m = rng.choice([1.0, 1 + 2.0 ** -52, 1.5, 2 - 2.0 ** -52], n)
        return sign * np.ldexp(m, rng.choice([-1023, -1022, -1021, -1020, 1019, 1020, 1021, 1022, 1023], n))
    return np.resize(np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, 1e-310, 2.2250738585072014e-308,
                               1.7976931348623157e308, 1.0, -1.0, 3.0, 1e-200]), n)


KINDS = ("wide", "window", "powers", "reciprocal ends", "special")


@pytest.mark.parametrize("kind", KINDS)
def test_quotients(kind):
    rng = np.random.default_rng(12)
    a, b = operands(kind, rng, 40000), rng.permutation(operands(kind, rng, 40000))
    got = evaluate(a, b)
    with np.errstate(all="ignore"):
        np.testing.assert_array_equal(bits(got["div_rn"]), bits(a / b))


@pytest.mark.parametrize("kind", KINDS[:3])
def test_reciprocals(kind):
    """1/b rounded to nearest, and the one that is within 0.52 ulp (measured against the
    remainder 1 - b r, exact in integers), where 1/b is normal."""
    rng = np.random.default_rng(13)
    b = operands(kind, rng, 40000)
    b = b[(np.abs(b) > 1e-307) & (np.abs(b) < 1e307)]
    got = evaluate(np.ones_like(b), b)
    np.testing.assert_array_equal(bits(got["rcp_rn"]), bits(1.0 / b))
    m, e = np.frexp(np.abs(got["rcp"]))
    mb, eb = np.frexp(np.abs(b))
    R, B = (np.ldexp(m, 53)).astype(np.int64), (np.ldexp(mb, 53)).astype(np.int64)
    for r, s, x in zip(R[:20000].tolist(), (106 - e - eb)[:20000].tolist(), B[:20000].tolist()):
        assert abs((1 << s) - r * x) * 100 <= 52 * x      # |1/b - r| <= 0.52 units of r
    assert np.array_equal(np.signbit(got["rcp"]), np.signbit(b))


def test_reciprocal_square_root_and_special_operands():
    rng = np.random.default_rng(14)
    b = np.concatenate([np.abs(operands(k, rng, 5000)) for k in ("wide", "powers")])
    b = b[b >= 2.2250738585072014e-308]
    got = evaluate(b, b)["rsqrt"]
    m, e = np.frexp(got)
    mb, eb = np.frexp(b)
    R, B = np.ldexp(m, 53).astype(np.int64), np.ldexp(mb, 53).astype(np.int64)
    for r, x, k in zip(R.tolist(), B.tolist(), (159 - 2 * e - eb).tolist()):
        # 1/sqrt(b) between r - 0.52 and r + 0.52 units: (100 r -+ 52)^2 x against 10^4 2^k
        assert (100 * r - 52) ** 2 * x <= 10 ** 4 << k <= (100 * r + 52) ** 2 * x
    # out of line, by the FP64 forms: their estimates flush subnormals to zero, and one
    # step from an infinite or zero estimate gives NaN (an infinity where it cancels)
    s = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, -1.0, 1e-310, 5e-324])
    got = evaluate(s, s)
    assert np.isnan(got["rsqrt"][:6]).all() and np.isinf(got["rsqrt"][6:]).all()
    assert np.isnan(got["rcp"][[0, 1, 2, 3, 4, 6, 7]]).all() and got["rcp"][5] == -1.0
