"""The work that is timed: what a user of the framework has it do, at the sizes
of its own set-ups, tests and benchmark.

Every case is one pass through the public entry points (`runtime.Simulation`
and the C ABI of include/mlh.h, or one of the batch functions of `runtime`).
"""
from __future__ import annotations

import ctypes
import math
from dataclasses import replace

import numpy as np
import torch

from meshlesshydro_gb300 import ic, runtime
from meshlesshydro_gb300.config import MFVConfig

STATE = ("x", "y", "z", "vx", "vy", "vz", "m", "u")


def listed():
    return [
        # one step of the smallest set-up of the test suite: launches and latency
        {"name": "kh24", "kind": "run", "setup": "kh", "n_side": 24, "steps": 1},
        # the reference's 2D test case (100 x 100), advanced to the next dump
        {"name": "kh100", "kind": "run", "setup": "kh", "n_side": 100, "steps": 8},
        # a finer 2D run with another adiabatic index (the general Riemann solver)
        {"name": "kh317_gamma14", "kind": "run", "setup": "kh", "n_side": 317, "steps": 2, "gamma": 1.4},
        # the reference's 3D test case: a blast in an open box, an odd lattice
        {"name": "sedov33_open", "kind": "run", "setup": "sedov", "n_side": 33, "steps": 3, "periodic": False},
        # the same in a periodic box, the ordinary 3D size
        {"name": "sedov64", "kind": "run", "setup": "sedov", "n_side": 64, "steps": 2},
        # the headline workload of bench.py, its largest single simulation
        {"name": "sedov128", "kind": "run", "setup": "sedov", "n_side": 128, "steps": 2},
        # many strong shocks, steps replayed as a CUDA graph
        {"name": "blasts48_graph", "kind": "run", "setup": "blasts", "n_side": 48, "steps": 3, "graph": True},
        # per-particle smoothing lengths
        {"name": "adaptive61", "kind": "run", "setup": "sedov", "n_side": 61, "steps": 2, "adaptive_h": True},
        # an ensemble of uneven 2D runs advanced together, as bench.py does
        {"name": "ensemble64_graph", "kind": "ensemble", "members": 64, "n_min": 2500, "n_max": 40000, "steps": 2},
        # a batch of Riemann problems through the host call (the Riemann class)
        {"name": "faces_250k", "kind": "faces", "dim": 3, "n": 250007},
        # the star-pressure network: prediction, and one batch's loss and gradient
        {"name": "infer_300k", "kind": "infer", "n": 300001},
        {"name": "grad_8k", "kind": "grad", "n": 8192},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["kh", "kh", "sedov", "sedov", "sedov", "blasts", "adaptive", "ensemble", "faces", "infer",
                       "grad"])
    if kind == "kh":
        return {"kind": "run", "setup": "kh", "n_side": _log_int(rng, 20, 600), "steps": rng.randint(1, 8),
                "gamma": rng.choice([5.0 / 3.0, 5.0 / 3.0, 1.4]), "graph": rng.random() < 0.3}
    if kind == "sedov":
        return {"kind": "run", "setup": "sedov", "n_side": _log_int(rng, 10, 120), "steps": rng.randint(1, 2),
                "periodic": rng.random() < 0.6, "graph": rng.random() < 0.3}
    if kind == "blasts":
        return {"kind": "run", "setup": "blasts", "n_side": _log_int(rng, 18, 72), "steps": rng.randint(1, 3),
                "graph": rng.random() < 0.5}
    if kind == "adaptive":
        return {"kind": "run", "setup": "sedov", "n_side": _log_int(rng, 12, 80), "steps": rng.randint(1, 2),
                "adaptive_h": True}
    if kind == "ensemble":
        lo = _log_int(rng, 600, 6000)
        return {"kind": "ensemble", "members": _log_int(rng, 3, 64), "n_min": lo, "n_max": 6 * lo,
                "steps": rng.randint(1, 3)}
    if kind == "faces":
        return {"kind": "faces", "dim": rng.choice([2, 3]), "n": _log_int(rng, 100, 500000)}
    if kind == "infer":
        return {"kind": "infer", "n": _log_int(rng, 500, 1000000)}
    return {"kind": "grad", "n": _log_int(rng, 500, 100000)}


# ------------------------------------------------------------------ inputs


def _member_sides(case):
    """Lattice sides of the members: particle counts spread evenly over their logarithm."""
    lo, hi = math.log(case["n_min"]), math.log(case["n_max"])
    at = [(7 * q % case["members"] + 0.5) / case["members"] for q in range(case["members"])]
    return [int(round(math.exp(0.5 * (lo + (hi - lo) * a)))) for a in at]


def _particles(case, seed):
    """Initial conditions and configuration of a run; a list of sets for an ensemble."""
    if case["kind"] == "ensemble":
        rng = np.random.default_rng(seed)
        sets = [ic.kelvin_helmholtz(n_side=k, seed=seed * 1009 + q, amplitude=float(rng.uniform(0.005, 0.05)))
                for q, k in enumerate(_member_sides(case))]
        return sets, MFVConfig.kelvin_helmholtz(sets[0])
    gamma = case.get("gamma", 5.0 / 3.0)
    if case["setup"] == "kh":
        p = ic.kelvin_helmholtz(n_side=case["n_side"], seed=seed, gamma=gamma)
        return p, MFVConfig.kelvin_helmholtz(p)
    periodic = case.get("periodic", True)
    if case["setup"] == "blasts":
        # an energy that leaves every state positive for any seed (blasts of
        # about 600 times the background's pressure)
        p = ic.multi_blast(n_side=case["n_side"], n_blasts=16, seed=seed, energy=0.005)
    else:
        p = ic.sedov(n_side=case["n_side"], seed=seed, periodic=periodic)
    cfg = MFVConfig.sedov(p, periodic=periodic)
    if case.get("adaptive_h"):
        # the search radius and the neighbour number of bench.py's adaptive workload
        cfg = replace(cfg, adaptive_h=True, n_ngb=32.0, kernel_size=1.25 * cfg.kernel_size)
    return p, cfg


def _pinned_view(n, dim):
    """Page-locked host arrays of a state and their mlh_particles_view."""
    host = {k: torch.zeros(n, dtype=torch.float64).pin_memory() for k in STATE if dim == 3 or k not in ("z", "vz")}
    view = runtime.ParticlesView()
    view.n = n
    for k, t in host.items():
        setattr(view, k, ctypes.cast(t.data_ptr(), ctypes.POINTER(ctypes.c_double)))
    return host, view


def _faces(case, seed):
    """Left and right states, frame velocities and face vectors: mostly weak
    jumps, as in a smooth flow, and one face in eight across a shock."""
    rng = np.random.default_rng(seed)
    n, d = case["n"], case["dim"]
    rho = np.exp(rng.normal(0.0, 0.5, n))
    p = np.exp(rng.normal(0.0, 1.0, n))
    strong = rng.random(n) < 0.125
    jump = np.where(strong, rng.normal(0.0, 3.0, n), rng.normal(0.0, 0.05, n))
    v = rng.normal(0.0, 1.0, (n, d))
    c = np.sqrt(5.0 / 3.0 * p / rho)
    dv = rng.normal(0.0, 1.0, (n, d)) * (np.where(strong, 0.5, 0.05) * c)[:, None]
    wi = np.column_stack([rho, p, v])
    wj = np.column_stack([rho * np.exp(0.4 * jump), p * np.exp(jump), v + dv])
    return wi, wj, rng.normal(0.0, 0.3, (n, d)), rng.normal(0.0, 1e-3, (n, d))


def _network(case, seed):
    rng = np.random.default_rng(seed)
    n = case["n"]
    lp = np.abs(rng.normal(0.0, 3.0, n))
    lr = 0.4 * lp + rng.normal(0.0, 0.3, n)
    x = np.column_stack([lr, rng.normal(-0.5, 0.7, n), lp, 0.5 * (lp - lr)]).astype(np.float32)
    t = (0.1 * rng.normal(0.0, 1.0, n) + 0.02 * lp).astype(np.float32)
    return runtime.pstar_init(seed), x, t


def prepare(case, seed):
    if case["kind"] == "faces":
        return {"kind": "faces", "args": _faces(case, seed)}
    if case["kind"] in ("infer", "grad"):
        w, x, t = _network(case, seed)
        return {"kind": case["kind"], "w": w, "x": x, "t": t}
    p, cfg = _particles(case, seed)
    if case["kind"] == "ensemble":
        sim = runtime.Simulation(cfg, members=p)
        p = ic.concatenate(p)
    else:
        sim = runtime.Simulation(cfg, p)
    if case["kind"] == "ensemble" or case.get("graph"):
        sim.set_graph_mode(True)
    src, src_view = _pinned_view(p.n, p.dim)
    for k in src:
        src[k].copy_(torch.from_numpy(getattr(p, k)))
    dst, dst_view = _pinned_view(p.n, p.dim)
    return {"kind": "run", "sim": sim, "steps": case["steps"], "src": src, "src_view": src_view, "dst": dst,
            "dst_view": dst_view}


def run(state):
    if state["kind"] == "faces":
        return runtime.riemann_fluxes(*state["args"])
    if state["kind"] == "infer":
        return runtime.pstar_infer(state["w"], state["x"])
    if state["kind"] == "grad":
        return runtime.pstar_grad(state["w"], state["x"], state["t"])
    # load a state, advance it to the next dump, read it back
    sim = state["sim"]
    sim.L.mlh_set_fields(sim.h, ctypes.byref(state["src_view"]))
    stats = sim.step(state["steps"], check=False)
    sim.L.mlh_get_fields(sim.h, ctypes.byref(state["dst_view"]))
    return {"state": state["dst"], "dt": stats.dt, "steps": stats.steps}


# ------------------------------------------------------------------ work

# FP64 operations of one step per particle: of the step's arithmetic with about
# 32 neighbours in 3D and 20 in 2D (bench.py's count for 3D)
_FLOPS = {2: 6.0e3, 3: 12.7e3}


def work(case):
    if case["kind"] == "faces":
        nv, d = case["dim"] + 2, case["dim"]
        return {"bytes": case["n"] * (8.0 * (3 * nv + 2 * d) + 4), "flops": 250.0 * case["n"]}
    if case["kind"] == "infer":
        return {"bytes": 20.0 * case["n"] + 4.0 * 8705, "flops": 17024.0 * case["n"]}
    if case["kind"] == "grad":
        return {"bytes": 20.0 * case["n"] + 8.0 * 8705, "flops": 3 * 17024.0 * case["n"]}
    if case["kind"] == "ensemble":
        n, d = sum(k * k for k in _member_sides(case)), 2
    else:
        d = 2 if case["setup"] == "kh" else 3
        n = case["n_side"] ** d
    # the state in and out of every step
    return {"bytes": 16.0 * (6 if d == 2 else 8) * n * case["steps"], "flops": _FLOPS[d] * n * case["steps"]}


# ------------------------------------------------------------------ exact results


def exact(case, seed):
    """The same results in 64 bits from plain numpy and torch."""
    if case["kind"] == "faces":
        wi, wj, vf, a = _faces(case, seed)
        return _exact_fluxes(wi, wj, vf, a, 5.0 / 3.0), None, None
    if case["kind"] in ("infer", "grad"):
        w, x, t = _network(case, seed)
        return _exact_network(w, x, t, case["kind"] == "grad")
    if case["kind"] == "ensemble" or case.get("adaptive_h"):
        return None
    if case["n_side"] ** (2 if case["setup"] == "kh" else 3) * case["steps"] > 120000:
        return None
    p, cfg = _particles(case, seed)
    s = {k: np.array(getattr(p, k)) for k in STATE}
    for _ in range(case["steps"]):
        dt = _exact_step(s, cfg)
    return {"state": {k: v for k, v in s.items() if p.dim == 3 or k not in ("z", "vz")}, "dt": dt, "steps": None}


def _exact_network(w, x, t, backward):
    w = torch.from_numpy(w).double().requires_grad_(backward)
    sizes = [(64, 4), (64,), (64, 64), (64,), (64, 64), (64,), (1, 64), (1,)]
    parts, at = [], 0
    for s in sizes:
        parts.append(w[at:at + math.prod(s)].reshape(s))
        at += math.prod(s)
    h = torch.from_numpy(x).double()
    for k in range(0, 6, 2):
        h = torch.nn.functional.silu(h @ parts[k].T + parts[k + 1])
    y = (h @ parts[6].T + parts[7])[:, 0]
    if not backward:
        return y
    loss = ((y - torch.from_numpy(t).double()) ** 2).mean()
    loss.backward()
    return float(loss.detach()), w.grad


def _riemann(g, rl, ul, pl, rr, ur, pr):
    """Exact Riemann solution sampled at x/t = 0 (Toro, chapter 4)."""
    with np.errstate(all="ignore"):
        cl, cr = np.sqrt(g * pl / rl), np.sqrt(g * pr / rr)
        z = (g - 1) / (2 * g)
        p = ((cl + cr - 0.5 * (g - 1) * (ur - ul)) / (cl / pl ** z + cr / pr ** z)) ** (1 / z)

        def f(p, r, pk, c):
            a, b = 2 / ((g + 1) * r), (g - 1) / (g + 1) * pk
            q = np.sqrt(a / (p + b))
            rare = p <= pk
            val = np.where(rare, 2 * c / (g - 1) * ((p / pk) ** z - 1), (p - pk) * q)
            der = np.where(rare, (p / pk) ** (z - 1) / (r * c), (1 - 0.5 * (p - pk) / (b + p)) * q)
            return val, der

        for _ in range(40):
            fl, dl = f(p, rl, pl, cl)
            fr, dr = f(p, rr, pr, cr)
            q = p - (fl + fr + ur - ul) / (dl + dr)
            q = np.where(q > 0, q, 1e-12 * np.maximum(pl, pr))
            done = np.max(np.abs(q - p) / (q + p)) < 1e-15
            p = q
            if done:
                break
        fl, fr = f(p, rl, pl, cl)[0], f(p, rr, pr, cr)[0]
        us = 0.5 * (ul + ur) + 0.5 * (fr - fl)
        right = us < 0
        s = np.where(right, -1.0, 1.0)          # the right side as the mirrored left side
        r, u, pk, c = np.where(right, rr, rl), s * np.where(right, ur, ul), np.where(right, pr, pl), np.where(right, cr, cl)
        v = s * us
        pm = p / pk
        g6 = (g - 1) / (g + 1)
        shock = p > pk
        sl = u - c * np.sqrt((g + 1) / (2 * g) * pm + z)
        head, tail = u - c, v - c * pm ** z
        cf = 2 / (g + 1) * (c + 0.5 * (g - 1) * u)
        fan = ~shock & (head < 0) & (tail >= 0)
        outside = np.where(shock, sl >= 0, head >= 0)
        rho = np.where(shock, r * (pm + g6) / (pm * g6 + 1), r * pm ** (1 / g))
        rho = np.where(fan, r * (cf / c) ** (2 / (g - 1)), rho)
        pres = np.where(fan, pk * (cf / c) ** (1 / z), p)
        vel = np.where(fan, cf, v)
        return (np.where(outside, r, rho), s * np.where(outside, u, vel), np.where(outside, pk, pres), right)


def _exact_fluxes(wi, wj, vf, a, g):
    """[mass, energy, momentum] through the faces a, in the lab frame."""
    hat = a / np.sqrt((a * a).sum(1))[:, None]
    ui, uj = (hat * wi[:, 2:]).sum(1), (hat * wj[:, 2:]).sum(1)
    rho, u, p, right = _riemann(g, wi[:, 0], ui, wi[:, 1], wj[:, 0], uj, wj[:, 1])
    v = np.where(right[:, None], wj[:, 2:], wi[:, 2:]) + (u - np.where(right, uj, ui))[:, None] * hat
    av = (a * v).sum(1)
    lab = v + vf
    mom = (rho * av)[:, None] * lab + p[:, None] * a
    energy = av * (p / (g - 1) + 0.5 * rho * (lab * lab).sum(1)) + p * (a * lab).sum(1)
    return np.column_stack([rho * av, energy, mom])


def _pairs(x, h, lo, hi, periodic):
    """All pairs closer than h, sorted by i: i, j, x_j - x_i, and whether j is a periodic image."""
    n, d = x.shape
    cells = np.maximum(np.floor((hi - lo) / h).astype(int), 1)
    at = np.clip(np.floor((x - lo) / ((hi - lo) / cells)).astype(int), 0, cells - 1)
    stride = np.concatenate([[1], np.cumprod(cells)[:-1]])
    order = np.argsort(at @ stride, kind="stable")
    start = np.searchsorted((at @ stride)[order], np.arange(cells.prod() + 1))
    found = []
    for off in np.ndindex(*(3,) * d):
        to = at + (np.array(off) - 1)
        wrap = np.floor_divide(to, cells)
        ok = np.ones(n, bool) if periodic else (wrap == 0).all(1)
        cell = (to - wrap * cells) @ stride
        b, e = start[cell], start[cell + 1]
        i = np.nonzero(ok)[0]
        cnt = (e - b)[i]
        ii = np.repeat(i, cnt)
        jj = order[np.repeat(b[i], cnt) + np.arange(cnt.sum()) - np.repeat(np.cumsum(cnt) - cnt, cnt)]
        dx = x[jj] + wrap[ii] * (hi - lo) - x[ii]
        image = (wrap[ii] != 0).any(1)
        keep = ((dx * dx).sum(1) < h * h) & (image | (ii != jj))
        found.append((ii[keep], jj[keep], dx[keep], image[keep]))
    i, j, dx, image = (np.concatenate(v) for v in zip(*found))
    o = np.argsort(i, kind="stable")
    return i[o], j[o], dx[o], image[o]


def _limit_pair(phi0, own, at_face, diff, below, psi1, psi2):
    """The pairwise limiter of one side of a face."""
    ad = np.abs(diff)
    shifted = np.where(below, own - psi1 * ad, own + psi1 * ad)
    with np.errstate(all="ignore"):
        damped = own / (1 + psi1 * ad / np.abs(own))
    bound = np.where((shifted >= 0) == (own >= 0), shifted, np.where(own == 0, 0.0, damped))
    low = np.maximum(bound, np.minimum(phi0, at_face + psi2 * ad))
    high = np.minimum(bound, np.maximum(phi0, at_face - psi2 * ad))
    return np.where(diff == 0, own, np.where(below, low, high))


def _exact_step(s, cfg):
    """One step of the scheme in place on the state s; returns its dt."""
    d, h, g = cfg.dim, cfg.kernel_size, cfg.gamma
    names = STATE[:d], STATE[3:3 + d]
    x, v = (np.stack([s[k] for k in ks], 1) for ks in names)
    m, u, n = s["m"], s["u"], len(s["m"])
    lo, hi = (np.array(cfg.box_lo[:d]), np.array(cfg.box_hi[:d])) if cfg.periodic else (x.min(0), x.max(0))
    i, j, dx, image = _pairs(x, h, lo, hi, cfg.periodic)
    r = np.sqrt((dx * dx).sum(1))
    w = ic.cubic_spline(r, h, d)

    def sums(a):
        return np.bincount(i, a, minlength=n)

    omega = sums(w) + ic.cubic_spline(np.zeros(1), h, d)[0]
    rho = m * omega
    pres = (g - 1) * rho * u
    c = np.sqrt(g * pres / rho)
    real = ~image
    vs = c[i] + c[j] - np.minimum(0, ((v[i] - v[j]) * -dx).sum(1) / r)
    dt = cfg.cfl * h / vs[real].max()
    wdx = dx * w[:, None]
    e = np.stack([np.stack([sums(dx[:, a] * wdx[:, b]) for b in range(d)], 1) for a in range(d)], 1)
    psi = np.einsum("pab,pb->pa", np.linalg.inv(e)[i], wdx)
    # fields in the order rho, P, v; their gradients, limited
    f = np.column_stack([rho, pres, v])
    first = np.searchsorted(i, np.arange(n))
    grad = np.empty((n, d + 2, d))
    tiny, huge = np.finfo(float).tiny, np.finfo(float).max
    for k in range(d + 2):
        df = f[j, k] - f[i, k]
        gk = np.stack([sums(df * psi[:, a]) for a in range(d)], 1)
        mid = f[i, k] + 0.5 * (gk[i] * dx).sum(1)
        hi_n, lo_n = np.maximum(np.maximum.reduceat(f[j, k], first), tiny), np.minimum(np.minimum.reduceat(f[j, k], first), huge)
        hi_m, lo_m = np.maximum(np.maximum.reduceat(mid, first), tiny), np.minimum(np.minimum.reduceat(mid, first), huge)
        with np.errstate(all="ignore"):
            top, bottom = np.abs((hi_n - f[:, k]) / (hi_m - f[:, k])), np.abs((f[:, k] - lo_n) / (f[:, k] - lo_m))
        scale = np.where((bottom <= top) & (cfg.beta * bottom < 1), bottom,
                         np.where((top <= bottom) & (cfg.beta * top < 1), top, 1.0))
        grad[:, k] = gk * scale[:, None]
    # faces i < j: the face vector needs the pair from the other side as well
    key = i.astype(np.int64) * n + j
    back = np.argsort(key)[np.searchsorted(np.sort(key), j.astype(np.int64) * n + i)]
    q = np.nonzero(j > i)[0]
    fi, fj, d2, im = i[q], j[q], 0.5 * dx[q], image[q]
    area = psi[q] / omega[fi][:, None] - psi[back[q]] / omega[fj][:, None]
    frame = 0.5 * (v[fi] + v[fj])
    left, right = f[fi].copy(), f[fj].copy()
    left[:, 2:] -= frame
    right[:, 2:] -= frame
    if cfg.pairwise_limiter:
        base = left.copy(), right.copy()
    left += np.einsum("pka,pa->pk", grad[fi], d2)
    right -= np.einsum("pka,pa->pk", grad[fj], d2)
    if cfg.pairwise_limiter:
        diff = base[0] - base[1]
        lim_l = _limit_pair(left, base[0], base[0] - 0.5 * diff, diff, diff < 0, cfg.psi1, cfg.psi2)
        lim_r = _limit_pair(right, base[1], base[1] + 0.5 * diff, -diff, diff > 0, cfg.psi1, cfg.psi2)
        left, right = np.where(im[:, None], left, lim_l), np.where(im[:, None], right, lim_r)
    # half a step of each particle's own evolution, seen from the moving face
    div = sum(grad[:, 2 + a, a] for a in range(d))
    src = np.column_stack([rho * div, g * pres * div, grad[:, 1] / rho[:, None]])
    ti = src + np.einsum("pka,pa->pk", grad, v)
    left -= 0.5 * dt * (ti[fi] - np.einsum("pka,pa->pk", grad[fi], frame))
    seen = np.repeat(frame[:, None, :], d + 2, 1)
    if d == 3:      # vx and vy of side j are advected with the vz of side i
        seen[:, 2:4, 2] -= (v[fi, 2] - v[fj, 2])[:, None]
    right -= 0.5 * dt * (ti[fj] - np.einsum("pka,pka->pk", grad[fj], seen))
    flux = _exact_fluxes(left, right, frame, area, g)
    total = np.stack([np.bincount(fi, flux[:, k], minlength=n) - np.bincount(fj, flux[:, k], minlength=n)
                      for k in range(d + 2)], 1)
    energy = m * (u + 0.5 * (v * v).sum(1)) - dt * total[:, 1]
    mom = m[:, None] * v - dt * total[:, 2:]
    s["m"] = m - dt * total[:, 0]
    vn = mom / s["m"][:, None]
    s["u"] = energy / s["m"] - 0.5 * (vn * vn).sum(1)
    x = x + v * dt
    if cfg.periodic:
        x = np.where(x < lo, hi - (lo - x), np.where(x >= hi, lo + (x - hi), x))
    for k, name in enumerate(names[0]):
        s[name] = x[:, k]
    for k, name in enumerate(names[1]):
        s[name] = vn[:, k]
    return float(dt)
