"""The slope limiter's single-precision filter with gradients in units of their own
size: the float32 arithmetic of the gradients kernel restated, its bound and its
candidates checked against the FP64 values, for gradients and fields far outside the
range of single precision as well."""
import numpy as np

f32 = np.float32
EPS32, U64 = f32(2.0 ** -24), f32(2.0 ** -53)
AS_IS = 896


def trunc_f32(x, base):
    """x 2^(896 - base), sign, exponent and top 23 mantissa bits; 0 below 2^-126."""
    b = np.asarray(x, np.float64).view(np.uint64)
    m = ((b & np.uint64(0x7FFFFFFFFFFFFFFF)) >> np.uint64(29)).astype(np.int64) - (base << 23)
    bits = np.where(m < (1 << 23), 0, np.minimum(m, 255 << 23)).astype(np.uint32)
    return (bits | ((b >> np.uint64(63)).astype(np.uint32) << np.uint32(31))).view(f32)


def base_of(g):
    e = int((np.abs(np.asarray(g, np.float64)).view(np.uint64) >> np.uint64(52)).max())
    return max(e - 127, 0)


def test_rebased_truncation():
    rng = np.random.default_rng(0)
    x = rng.standard_normal(5000) * 10.0 ** rng.uniform(-300, 300, 5000)
    for v in x:
        b = base_of([v])
        t = float(trunc_f32([v], b)[0])
        exact = np.ldexp(v, 896 - b)
        assert (1 <= abs(t) < 2 or b == 0) and abs(t - exact) <= 2.0 ** -23 * abs(exact) and abs(t) <= abs(exact)


def test_candidates_hold_the_extrema_at_every_scale():
    rng = np.random.default_rng(1)
    kept = 0
    for t in range(6000):
        D, n = 2 + t % 2, int(rng.integers(1, 60))
        d = (rng.random((n, D)) * 2 - 1) * 10.0 ** rng.integers(-6, 20)
        if t % 5 == 0:
            d = np.round(d / np.abs(d).max() * 2) / 2 * np.abs(d).max()
        g = rng.standard_normal(D) * 10.0 ** rng.integers(-250, 250) * rng.choice([1.0, 1e-9, 1e-30], D)
        fi = rng.standard_normal() * np.abs(g).max() * np.abs(d).max() * 10.0 ** rng.integers(-3, 12)
        fij = np.full(n, fi)
        for a in range(D):
            fij = fij + g[a] * d[:, a]
        b = base_of(g)
        gf, df, fa = trunc_f32(g, b), trunc_f32(d, AS_IS), abs(trunc_f32([fi], b)[0]) * (f32(1) + f32(4) * EPS32)
        q = (gf[0] * df[:, 0]).astype(f32)
        for a in range(1, D):
            q = (q + (gf[a] * df[:, a]).astype(f32)).astype(f32)
        R = f32(np.abs(df).max()) * (f32(1) + f32(4) * EPS32) + f32(1e-30)
        S = f32(np.abs(gf).sum())
        if not (S * R < 1e36 and fa < 1e36):
            continue
        B = f32(16) * EPS32 * S * R + f32(12) * U64 * (fa + S * R) + f32(1e-36)
        unit = np.ldexp(1.0, b - 896) if b - 896 > -1000 else np.ldexp(1.0, -1000)
        assert np.all(np.abs((fij - fi) / unit - q.astype(np.float64)) <= B)
        cand = (q >= q.max() - f32(2) * B) | (q <= q.min() + f32(2) * B)
        assert np.any(fij[cand] == fij.max()) and np.any(fij[cand] == fij.min())
        kept += 1
    assert kept > 5000


def test_signal_speed_bound_in_units_of_kernel_size():
    rng = np.random.default_rng(2)
    used = 0
    for t in range(6000):
        D, n = 2 + t % 2, int(rng.integers(1, 40))
        h = 10.0 ** rng.uniform(-200, 200)
        d = (rng.random((n, D)) * 2 - 1) * h / np.sqrt(D) * 10.0 ** -rng.integers(0, 9)
        if t % 7 == 0:
            d[::2, 0] = rng.choice([0.0, 1e-45 * h, -1e-40 * h, 1e-60 * h], d[::2, 0].shape)
        r = np.sqrt(np.sum((d / h) ** 2, axis=1)) * h
        scale = 10.0 ** rng.integers(-26, 26)
        vi = rng.standard_normal(D) * scale
        vj = vi + rng.standard_normal((n, D)) * scale * (0.0 if t % 9 == 0 else 1.0)
        ci, cj = abs(rng.standard_normal()) * scale, np.abs(rng.standard_normal(n)) * scale
        dv = np.sum((vi - vj) * -(d / h), axis=1)
        with np.errstate(all="ignore"):
            vs = np.where(dv < 0, ci + cj - dv / (r / h), ci + cj)
        df, vif, vjf = trunc_f32(d, base_of([h])), vi.astype(f32), vj.astype(f32)
        with np.errstate(all="ignore"):
            w = (vif - vjf).astype(f32)
            dvd = np.sum((w * df).astype(f32), axis=1, dtype=f32)
            rf = np.sqrt(np.sum((df * df).astype(f32), axis=1, dtype=f32)).astype(f32)
            T = np.where(dvd > 0, (dvd / rf).astype(f32), f32(0))
            vsf = (f32(ci) + cj.astype(f32) + T).astype(f32)
            V = (np.abs(vif).sum() + np.abs(vjf).sum(axis=1)).astype(f32)
            B = f32(2) * EPS32 * (f32(2) * (f32(ci) + cj.astype(f32)) + f32(2) * vsf + f32(16) * V)
        ok = (rf > f32(1e-12)) & (rf < f32(1e15)) & (B > f32(1e-31)) & (B < f32(1e30))
        assert np.all(np.abs(vsf.astype(np.float64) - vs)[ok] <= B[ok]), t
        used += ok.mean()
    assert used > 5500
