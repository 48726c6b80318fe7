"""The single-precision filters of the gradients kernel on truncated offsets: the
float32 arithmetic restated, and its bounds checked against the FP64 values they
have to contain (random offsets and gradients, lattice ties, zeros, tiny offsets
that flush to zero)."""
import numpy as np

f32 = np.float32
EPS32, U64 = f32(2.0 ** -24), f32(2.0 ** -53)


def trunc_f32(x):
    """The double's sign, exponent and top 23 mantissa bits; zero below 2^-126."""
    b = np.asarray(x, np.float64).view(np.uint64)
    mag = b & np.uint64(0x7FFFFFFFFFFFFFFF)
    m = (mag >> np.uint64(29)).astype(np.int64) - (896 << 23)
    bits = np.where(m < (1 << 23), 0, np.minimum(m, 255 << 23)).astype(np.uint32)
    return (bits | ((b >> np.uint64(63)).astype(np.uint32) << np.uint32(31))).view(f32)


def offsets(rng, n, D, t):
    d = (rng.random((n, D)) * 2 - 1) * 10.0 ** rng.integers(-6, 3)
    if t % 5 == 0:
        d = np.round(d / np.abs(d).max() * 2) / 2 * np.abs(d).max()     # a lattice: ties and zeros
    if t % 7 == 0:
        d[:: 2, 0] = rng.choice([0.0, 1e-45, -1e-40, 1e-310], d[:: 2, 0].shape)
    return d


def test_trunc_f32_error():
    rng = np.random.default_rng(0)
    x = rng.standard_normal(20000) * 10.0 ** rng.uniform(-60, 30, 20000)
    t = trunc_f32(x).astype(np.float64)
    assert np.all(np.abs(t - x) <= np.maximum(2.0 ** -23 * np.abs(x), 2.0 ** -126))
    assert np.all(np.abs(t) <= np.abs(x))


def test_limiter_extrema_are_candidates():
    rng = np.random.default_rng(1)
    for D in (2, 3):
        for t in range(3000):
            n = int(rng.integers(1, 60))
            d = offsets(rng, n, D, t)
            g = rng.standard_normal(D) * 10.0 ** rng.integers(-4, 4) * (0.0 if t % 11 == 0 else 1.0)
            fi = rng.standard_normal() * 10.0 ** rng.integers(-4, 4)
            fij = np.full(n, fi)
            for a in range(D):
                fij = fij + g[a] * d[:, a]
            gf, df = g.astype(f32), trunc_f32(d)
            q = (gf[0] * df[:, 0]).astype(f32)
            for a in range(1, D):
                q = (q + (gf[a] * df[:, a]).astype(f32)).astype(f32)
            R = f32(np.abs(df).max()) * (f32(1) + f32(4) * EPS32) + f32(1e-30)
            S = f32(np.abs(gf).sum())
            B = f32(16) * EPS32 * S * R + f32(12) * U64 * (f32(abs(fi)) + S * R) + f32(1e-36)
            assert np.all(np.abs(fij - (fi + q.astype(np.float64))) <= B), (D, t)
            cand = (q >= q.max() - f32(2) * B) | (q <= q.min() + f32(2) * B)
            assert np.any(fij[cand] == fij.max()) and np.any(fij[cand] == fij.min()), (D, t)


def test_signal_speed_bound():
    rng = np.random.default_rng(2)
    for D in (2, 3):
        for t in range(3000):
            n = int(rng.integers(1, 40))
            d = offsets(rng, n, D, t)
            r = np.sqrt(np.sum(d * d, axis=1))
            scale = 10.0 ** rng.integers(-3, 3)
            vi = rng.standard_normal(D) * scale
            vj = vi + rng.standard_normal((n, D)) * scale * (0.0 if t % 9 == 0 else 1.0)
            ci, cj = abs(rng.standard_normal()) * scale, np.abs(rng.standard_normal(n)) * scale
            dv = np.sum((vi - vj) * -d, axis=1)
            with np.errstate(all="ignore"):
                vs = np.where(dv < 0, ci + cj - dv / r, ci + cj)
            df, vif, vjf = trunc_f32(d), vi.astype(f32), vj.astype(f32)
            w = (vif - vjf).astype(f32)
            dvd = np.sum((w * df).astype(f32), axis=1, dtype=f32)
            rf = np.sqrt(np.sum((df * df).astype(f32), axis=1, dtype=f32)).astype(f32)
            usable = (rf > f32(1e-15)) & (rf < f32(1e15))
            with np.errstate(all="ignore"):
                T = np.where(dvd > 0, (dvd / rf).astype(f32), f32(0))
            vsf = (f32(ci) + cj.astype(f32) + T).astype(f32)
            V = (np.abs(vif).sum() + np.abs(vjf).sum(axis=1)).astype(f32)
            B = f32(2) * EPS32 * (f32(2) * (f32(ci) + cj.astype(f32)) + f32(2) * vsf + f32(16) * V)
            assert np.all(np.abs(vsf.astype(np.float64) - vs)[usable] <= B[usable]), (D, t)
