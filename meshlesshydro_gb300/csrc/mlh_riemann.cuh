// Exact Riemann solver for an ideal gas on the device, one thread per face.
//
// Method: E. F. Toro, "Riemann Solvers and Numerical Methods for Fluid
// Dynamics", 3rd ed., ch. 4: Newton-Raphson on f(p) = fL(p) + fR(p) + du for
// the star pressure, two-rarefaction initial guess, sampling at x/t = 0.  The
// reference calls the third-party RiemannSolver.hpp for this step
// (demonstrator/src/Riemann.cpp:84-94), whose sources are not in its tree; this
// solver fixes the guess, the convergence test |dp| / p_mean <= tol and the
// sampling rules, the same choices as the CPU oracle.
#pragma once
#include "mlh_device.cuh"

namespace mlh {

struct RiemannConsts {
    double gamma, g1, g2, g3, g4, g5, g6, g7, inv_gamma, inv_gm1, tol;
    double tol_half;   // tol / 2 (exact): 2 |dp| <= tol s  <=>  |dp| <= (tol / 2) s
    double ig5;   // 1 / g5 = (gamma + 1) / 2
    double g6ig5; // g6 ig5 = (gamma - 1) / 2
    int max_iter;
    // 2 gamma / (gamma - 1) where it is 5 (gamma = 5/3) or 7 (gamma = 7/5), else
    // 0.  With N = 2 gamma / (gamma - 1): g1 = 1/N, g3 = N, g4 = N - 2 and
    // 1/gamma = (N - 2) g1, so every power in the solver is an N-th root or an
    // integer power (10^6 2D faces at gamma = 7/5: 322 us, with pow 3180 us)
    int root;
};

__host__ __device__ inline RiemannConsts make_riemann_consts(double gamma, double tol, int max_iter) {
    RiemannConsts c;
    c.gamma = gamma;
    c.g1 = (gamma - 1.) / (2. * gamma);
    c.g2 = (gamma + 1.) / (2. * gamma);
    c.g3 = 2. * gamma / (gamma - 1.);
    c.g4 = 2. / (gamma - 1.);
    c.g5 = 2. / (gamma + 1.);
    c.ig5 = (gamma + 1.) / 2.;
    c.g6ig5 = (gamma - 1.) / 2.;
    c.g6 = (gamma - 1.) / (gamma + 1.);
    c.g7 = (gamma - 1.) / 2.;
    c.inv_gamma = 1. / gamma;
    c.inv_gm1 = 1. / (gamma - 1.);
    c.tol = tol;
    c.tol_half = tol / 2.;
    c.max_iter = max_iter;
    c.root = 0;
    for (int n = 5; n <= 7; n += 2)
        if (fabs(1. / c.g1 - n) < 1e-12 && fabs(c.g4 - (n - 2)) < 1e-12) c.root = n;
    return c;
}

// f_K and f_K' (Toro eqs. 4.6, 4.7, 4.37); (p/pK)^(-(g+1)/(2g)) = (p/pK)^g1 / (p/pK).
__device__ __forceinline__ void pressure_fn(const RiemannConsts &c, double p, double rhoK, double pK, double cK,
                                            double &f, double &fd) {
    if (p <= pK) {
        double prat = p / pK;
        double q = pow(prat, c.g1);
        f = c.g4 * cK * (q - 1.);
        fd = q / (prat * rhoK * cK);
    } else {
        double ak = c.g5 / rhoK;
        double bk = c.g6 * pK;
        double qrt = sqrt(ak / (bk + p));
        f = (p - pK) * qrt;
        fd = (1. - .5 * (p - pK) / (bk + p)) * qrt;
    }
}

struct RiemannResult {
    double rho, u, p;
    double pstar;   // star-region pressure
    int flag;       // -1: left of the contact sampled, +1: right, 0: vacuum,
                    // 2: not solved (two-rarefaction guess above `defer_above`)
    int iters;      // Newton iterations (< 0: no convergence)
};

// Newton-Raphson from p0; returns iterations or -1.
__device__ __forceinline__ int newton_pstar(const RiemannConsts &c, double p0, double rhoL, double uL, double pL,
                                            double cL, double rhoR, double uR, double pR, double cR, double &pstar) {
    double pfloor = 1e-12 * (pL > pR ? pL : pR);
    double p = p0 > pfloor ? p0 : pfloor;
    double du = uR - uL;
    for (int it = 1; it <= c.max_iter; ++it) {
        double fL, fdL, fR, fdR;
        pressure_fn(c, p, rhoL, pL, cL, fL, fdL);
        pressure_fn(c, p, rhoR, pR, cR, fR, fdR);
        double pnew = p - (fL + fR + du) / (fdL + fdR);
        if (!(pnew > 0.)) pnew = pfloor;
        double change = 2. * fabs(pnew - p) / (pnew + p);
        p = pnew;
        if (change <= c.tol) { pstar = p; return it; }
    }
    pstar = p;
    return -1;
}

// Solve with the two-rarefaction guess (or `guess` when > 0, falling back to
// the two-rarefaction guess if Newton does not converge from it), then sample
// at S = 0 (Toro section 4.5).  With defer_above > 0 and no guess, a problem
// whose two-rarefaction guess exceeds defer_above returns unsolved (flag 2,
// pstar = that guess) for a second pass with a better guess.
__device__ inline RiemannResult riemann_exact(const RiemannConsts &c, double rhoL, double uL, double pL,
                                              double rhoR, double uR, double pR, double guess = -1.,
                                              double defer_above = 0.) {
    RiemannResult res;
    double cL = sqrt(c.gamma * pL / rhoL);
    double cR = sqrt(c.gamma * pR / rhoR);
    if (c.g4 * (cL + cR) <= uR - uL) {
        res.rho = 0.; res.u = 0.; res.p = 0.; res.pstar = 0.; res.flag = 0; res.iters = 0;
        return res;
    }
    double pstar;
    int it = -1;
    if (guess > 0.) it = newton_pstar(c, guess, rhoL, uL, pL, cL, rhoR, uR, pR, cR, pstar);
    if (it < 0) {
        double num = cL + cR - c.g7 * (uR - uL);
        double den = cL / pow(pL, c.g1) + cR / pow(pR, c.g1);
        double p0 = pow(num / den, c.g3);
        if (defer_above > 0. && !(guess > 0.) && p0 > defer_above) {
            res.rho = 0.; res.u = 0.; res.p = 0.; res.pstar = p0; res.flag = 2; res.iters = 0;
            return res;
        }
        int it2 = newton_pstar(c, p0, rhoL, uL, pL, cL, rhoR, uR, pR, cR, pstar);
        it = (guess > 0. && it2 >= 0) ? it2 + c.max_iter : it2;
        if (it2 < 0) it = -1;
    }
    res.iters = it;
    res.pstar = pstar;
    double fL, fdL, fR, fdR;
    pressure_fn(c, pstar, rhoL, pL, cL, fL, fdL);
    pressure_fn(c, pstar, rhoR, pR, cR, fR, fdR);
    double ustar = .5 * (uL + uR) + .5 * (fR - fL);
    double rho, u, p;
    if (0. <= ustar) {
        if (pstar <= pL) {
            double shl = uL - cL;
            if (0. <= shl) { rho = rhoL; u = uL; p = pL; }
            else {
                double cml = cL * pow(pstar / pL, c.g1);
                double stl = ustar - cml;
                if (0. > stl) { rho = rhoL * pow(pstar / pL, c.inv_gamma); u = ustar; p = pstar; }
                else {
                    double cf = c.g5 * (cL + c.g7 * uL);
                    u = cf;
                    rho = rhoL * pow(cf / cL, c.g4);
                    p = pL * pow(cf / cL, c.g3);
                }
            }
        } else {
            double pml = pstar / pL;
            double sl = uL - cL * sqrt(c.g2 * pml + c.g1);
            if (0. <= sl) { rho = rhoL; u = uL; p = pL; }
            else { rho = rhoL * (pml + c.g6) / (pml * c.g6 + 1.); u = ustar; p = pstar; }
        }
        res.flag = -1;
    } else {
        if (pstar > pR) {
            double pmr = pstar / pR;
            double sr = uR + cR * sqrt(c.g2 * pmr + c.g1);
            if (0. >= sr) { rho = rhoR; u = uR; p = pR; }
            else { rho = rhoR * (pmr + c.g6) / (pmr * c.g6 + 1.); u = ustar; p = pstar; }
        } else {
            double shr = uR + cR;
            if (0. >= shr) { rho = rhoR; u = uR; p = pR; }
            else {
                double cmr = cR * pow(pstar / pR, c.g1);
                double str = ustar + cmr;
                if (0. <= str) { rho = rhoR * pow(pstar / pR, c.inv_gamma); u = ustar; p = pstar; }
                else {
                    double cf = c.g5 * (cR - c.g7 * uR);
                    u = -cf;
                    rho = rhoR * pow(cf / cR, c.g4);
                    p = pR * pow(cf / cR, c.g3);
                }
            }
        }
        res.flag = 1;
    }
    res.rho = rho; res.u = u; res.p = p;
    return res;
}

// ---------------------------------------------------------------- fast path

// Comparison of non-negative doubles on the integer pipe: their bit patterns
// are ordered as the values.
__device__ __forceinline__ bool nn_le(double a, double b) { return __double_as_longlong(a) <= __double_as_longlong(b); }

// x < 0, false for NaN of either sign (dneg goes by the sign bit)
__device__ __forceinline__ bool below_zero(double x) {
    return (unsigned long long)__double_as_longlong(x) - 0x8000000000000001ull <= 0x7fefffffffffffffull;
}

// The multiplies, adds and fused multiply-adds of the fast path are written
// out (mulr, addr, subr, fma): left to the compiler, their fusing would depend
// on the basic blocks around them and so on the kernel that inlines the
// solver, whose variants have to give the same bits.

// x^N and x^(N-2) for N = 5, 7
template <int N>
__device__ __forceinline__ double pow_n(double x, double &xm2) {
    const double x2 = mulr(x, x), x3 = mulr(x2, x), x5 = mulr(x3, x2);
    if (N == 5) { xm2 = x3; return x5; }
    xm2 = x5;
    return mulr(x5, x2);
}

// Two-rarefaction estimate of p* (Toro eq. 4.46), the default starting point
// of both solvers; ROOT takes the roots of its gamma (0: any gamma).  Not
// positive when the states generate vacuum.
template <int ROOT>
__device__ __forceinline__ double two_rarefaction_guess(const RiemannConsts &k, double rhoL, double uL, double pL,
                                                        double rhoR, double uR, double pR) {
    const double cL = sqrt(k.gamma * pL / rhoL), cR = sqrt(k.gamma * pR / rhoR);
    const double num = cL + cR - k.g7 * (uR - uL);
    if (!(num > 0.)) return -1.;
    if (ROOT) {
        constexpr int N = ROOT ? ROOT : 5;
        const double t = fdiv(num, cL * rroot<N>(pL) + cR * rroot<N>(pR));
        double tm2;
        return pow_n<N>(t, tm2);
    }
    return pow(num / (cL / pow(pL, k.g1) + cR / pow(pR, k.g1)), k.g3);
}

// A side of the problem: a = 1 / A_K = rho / g5, b = B_K a (so that
// (B_K + p) / A_K = a p + b), C = c / gamma, g4c = g4 c.
struct RiemannSide {
    double rho, u, p, c, invp, C, a, b, g4c;
};

__device__ __forceinline__ RiemannSide make_side(const RiemannConsts &k, double rho, double u, double p) {
    RiemannSide s;
    s.rho = rho; s.u = u; s.p = p;
    const double rp = xmul(rho, p);
    // c = sqrt(gamma p / rho) = gamma p / sqrt(gamma p rho)
    s.c = xmul(xmul(k.gamma, p), frsqrt(xmul(k.gamma, rp)));
    s.invp = frcp(p);
    s.C = xmul(s.c, k.inv_gamma);     // pK / (rhoK cK) = cK / gamma: f' = (p/pK)^g1 C / p
    s.a = xmul(rho, k.ig5);
    s.b = xmul(rp, k.g6ig5);
    s.g4c = xmul(k.g4, s.c);
    return s;
}

// f_K, f_K' at p (1/p given); q = (p/pK)^g1 on the rarefaction branch
template <int N>
__device__ __forceinline__ void pressure_fn_root(const RiemannSide &s, double p, double invp, double &f, double &fd,
                                                 double &q, bool &rare) {
    if (nn_le(p, s.p)) {
        q = root<N>(xmul(p, s.invp));
        f = fma(s.g4c, q, -s.g4c);
        fd = xmul(xmul(q, s.C), invp);
        rare = true;
    } else {
        // qrt = sqrt(A_K / (B_K + p)) and t = 1 / (B_K + p) from one
        // reciprocal square root: qrt = 1/sqrt((B_K + p) / A_K), t = qrt^2 / A_K
        const double qrt = frsqrt(fma(s.a, p, s.b));
        // t / 2 = qrt^2 A_K^-1 / 2, halved through the operand (exact), so
        // that nothing on the iteration's dependency chain waits on it
        const double t2 = xmul(xmul(qrt, qrt), half_of(s.a));
        const double d = subr(p, s.p);
        f = mulr(d, qrt);
        fd = xmul(fma(-d, t2, 1.), qrt);
        q = 0.;
        rare = false;
    }
}

// Same solution as riemann_exact for N = 2 gamma / (gamma - 1) = 5 or 7 with
// cheaper arithmetic: N-th roots instead of pow, integer powers for g3, g4 and
// 1/gamma, f_K(p*) from the last Newton evaluation plus its derivative times
// the final (<= tol relative) step, which differs from re-evaluating f at p*
// by O(tol^2) relative, and sign and order tests, halvings, reciprocals, roots
// and most products on the integer pipe (mlh_intmath.cuh).  A product goes
// there (xmul) where both factors are positive in every physical state, so
// that its range test never fails; products that can be zero, and sums, stay
// on the FP64 pipe.
// first_iters > 0: when Newton from the two-rarefaction guess has not
// converged after that many steps, return unsolved (flag 2, pstar = the
// current iterate, iters = steps run); solving again with that iterate as
// `guess` continues the same iteration with the same arithmetic.
//
// Two mirror images keep the lanes of a warp on one branch (a warp issues
// every branch that any of its lanes takes, and on this GPU an FP64
// instruction costs the same with one active lane as with 32).  The Euler
// equations are symmetric under swapping the sides and negating the
// velocities: p* is unchanged and u* and the sampled velocity change sign.
// (1) Newton solves the problem with the lower pressure on the left (A) and
// the higher on the right (B).  It performs the same operations on the same
// operands as for the unsorted problem, with the two sides' terms added in
// the other order (IEEE addition commutes, and uR - uL is unchanged), so p*
// is the same double.  In the weak-wave faces that make up most of a step,
// p* lies between pL and pR: A is a shock and B a rarefaction in nearly
// every lane, where the unsorted problem splits each side's branch of
// pressure_fn_root at random.  (2) The solution is sampled at S = 0 by the
// left-side logic only: on the left state as given when the contact moves
// right (u* >= 0), on the mirror image of the right state otherwise.  Every
// speed of the mirrored sampling is the exact negation of the right-side
// speed it stands for, and the ties at zero are resolved as the right-side
// tests resolve them, so the sampled state is the one of the two-sided
// sampling (Toro section 4.5).
// State of the root solver between its phases: the sorted sides, the Newton
// iterate and, once converged, f_K(p*) and (p*/p_K)^(1/N).
struct RootSolve {
    RiemannSide A, B;
    double du, pfloor, p, fAs, fBs, qAs, qBs;
    int iters;   // Newton steps run (a restart from p_TR counts max_iter first); -1: no convergence
    int stage;   // 0 vacuum; 1 Newton done (finish next); 2 stopped unfinished; 3 strong shock deferred
    bool mir;
};

// p_TR (Toro eq. 4.46) of the sorted problem.
template <int N>
__device__ __forceinline__ double root_guess(const RiemannConsts &k, const RiemannSide &A, const RiemannSide &B,
                                             double csum, double du) {
    const double num = fma(-k.g7, du, csum);
    const double den = fma(A.c, rroot<N>(A.p), xmul(B.c, rroot<N>(B.p)));
    const double t = mulr(num, frcp(den));
    const double t2 = xmul(t, t), t4 = xmul(t2, t2);
    return N == 5 ? xmul(t4, t) : xmul(xmul(t4, t2), t);
}

// Newton from p0 (raised to the floor) on the sorted problem; with
// tried_guess, a start that does not converge is retried from p_TR.
// first_iters > 0 (not with tried_guess): stop unfinished after that many
// steps (stage 2, s.p the iterate).
template <int N>
__device__ __forceinline__ void riemann_root_newton(const RiemannConsts &k, RootSolve &s, double p0, bool tried_guess,
                                                int first_iters) {
    const RiemannSide &A = s.A, &B = s.B;
    const double du = s.du, pfloor = s.pfloor;
    double p = p0;
    int iters = -1, extra = 0;
    s.fAs = 0.; s.fBs = 0.; s.qAs = -1.; s.qBs = -1.;
    for (int attempt = 0; attempt < 2 && iters < 0; ++attempt) {
        if (attempt == 1) {
            if (!tried_guess) break;
            extra = k.max_iter;
            p0 = root_guess<N>(k, A, B, addr(A.c, B.c), du);
        }
        p = nn_le(p0, pfloor) ? pfloor : p0;
        for (int it = 1; it <= k.max_iter; ++it) {
            double invp = frcp(p);
            double fA, fdA, qA, fB, fdB, qB;
            bool rA, rB;
            pressure_fn_root<N>(A, p, invp, fA, fdA, qA, rA);
            pressure_fn_root<N>(B, p, invp, fB, fdB, qB, rB);
            double pnew = fma(-addr(addr(fA, fB), du), frcp(addr(fdA, fdB)), p);
            {   // !(pnew > 0): zero, negative or NaN (bit patterns)
                const long long pb = __double_as_longlong(pnew);
                if (pb <= 0 || pb > 0x7FF0000000000000ll) pnew = pfloor;
            }
            const double dp = subr(pnew, p);
            if (nn_le(abs_bits(dp), mulr(k.tol_half, addr(pnew, p)))) {
                s.fAs = fma(fdA, dp, fA);
                s.fBs = fma(fdB, dp, fB);
                const double rel = mulr(k.g1, mulr(dp, invp));
                s.qAs = rA ? fma(qA, rel, qA) : -1.;
                s.qBs = rB ? fma(qB, rel, qB) : -1.;
                p = pnew;
                iters = it;
                break;
            }
            p = pnew;
            if (first_iters > 0 && !tried_guess && it >= first_iters) {
                s.p = p; s.iters = it; s.stage = 2;
                return;
            }
        }
    }
    s.p = p;
    s.iters = iters < 0 ? -1 : iters + extra;
    s.stage = 1;
}

// Whether the root solver takes a problem.  At gamma = 7/5 only one with densities
// and pressures in 2^-400 .. 2^400 and finite velocities, where its products and
// roots stay normal; the rest (cold gas with p = 0 above all, and states that are
// no physical ones) goes to riemann_exact, as with any other gamma: the root solver
// calls a side without pressure a vacuum.  At gamma = 5/3 it takes every problem.
template <int N>
__device__ __forceinline__ bool root_takes(double rhoL, double uL, double pL, double rhoR, double uR, double pR) {
    if (N == 5) return true;
    auto off = [](double x) { return (uint32_t)__double2hiint(x) - (623u << 20) >= 800u << 20; };
    auto infinite = [](double x) { return ((uint32_t)__double2hiint(x) & 0x7fffffffu) >= 0x7ff00000u; };
    return !(off(rhoL) | off(pL) | off(rhoR) | off(pR) | infinite(uL) | infinite(uR));
}

// riemann_exact out of line, from scalars (a reference to a kernel's constants would
// be a copy on the stack)
static __device__ __noinline__ RiemannResult riemann_exact_call(double gamma, double tol, int max_iter, double rhoL,
                                                                double uL, double pL, double rhoR, double uR,
                                                                double pR) {
    return riemann_exact(make_riemann_consts(gamma, tol, max_iter), rhoL, uL, pL, rhoR, uR, pR);
}

// The sides, the vacuum test, the start (the given guess, or p_TR) and the
// Newton iteration of riemann_exact_root, up to its optional stops.
template <int N>
__device__ __forceinline__ RootSolve riemann_root_begin(const RiemannConsts &k, double rhoL, double uL, double pL,
                                                 double rhoR, double uR, double pR, double guess,
                                                 double defer_above, int first_iters) {
    RootSolve s;
    s.mir = dlt(pR, pL);
    const bool mir = s.mir;
    s.A = make_side(k, mir ? rhoR : rhoL, mir ? flip_if(uR, true) : uL, mir ? pR : pL);
    s.B = make_side(k, mir ? rhoL : rhoR, mir ? flip_if(uL, true) : uR, mir ? pL : pR);
    s.fAs = 0.; s.fBs = 0.; s.qAs = -1.; s.qBs = -1.; s.iters = 0; s.p = 0.;
    // the sorted problem's uB - uA, from the given velocities: flips on the
    // integer pipe would turn a NaN's sign, which the vacuum test's order reads
    s.du = subr(uR, uL);
    const double csum = addr(s.A.c, s.B.c);
    if (!dlt(s.du, xmul(k.g4, csum))) {         // g4 (cL + cR) <= uR - uL: vacuum
        s.stage = 0;
        return s;
    }
    s.pfloor = xmul(1e-12, s.B.p);              // 1e-12 max(pL, pR)
    double p0;
    const bool tried_guess = __double_as_longlong(guess) > 0;   // guess > 0 (-1: none)
    if (tried_guess) p0 = guess;
    else {
        p0 = root_guess<N>(k, s.A, s.B, csum, s.du);
        // defer_above > 0 and p0 > defer_above, on the keys (see riemann_exact)
        if (ord_key(defer_above) > 0 && dlt(defer_above, p0)) {
            s.p = p0; s.stage = 3;
            return s;
        }
    }
    riemann_root_newton<N>(k, s, p0, tried_guess, first_iters);
    return s;
}

// Continue a solve stopped unfinished (stage 2) from its iterate: the same
// iteration as restarting riemann_exact_root with the iterate as the guess.
template <int N>
__device__ __forceinline__ void riemann_root_continue(const RiemannConsts &k, RootSolve &s) {
    riemann_root_newton<N>(k, s, s.p, true, 0);
}

template <int N>
__device__ inline RiemannResult riemann_root_finish(const RiemannConsts &k, const RootSolve &s);

template <int N>
__device__ inline RiemannResult riemann_exact_root(const RiemannConsts &k, double rhoL, double uL, double pL,
                                               double rhoR, double uR, double pR, double guess = -1.,
                                               double defer_above = 0., int first_iters = 0) {
    const RootSolve s = riemann_root_begin<N>(k, rhoL, uL, pL, rhoR, uR, pR, guess, defer_above, first_iters);
    RiemannResult res;
    if (s.stage == 0) {
        res.rho = 0.; res.u = 0.; res.p = 0.; res.pstar = 0.; res.flag = 0; res.iters = 0;
        return res;
    }
    if (s.stage >= 2) {   // unfinished (the iterate) or deferred strong shock (p_TR)
        res.rho = 0.; res.u = 0.; res.p = 0.; res.pstar = s.p; res.flag = 2; res.iters = s.stage == 2 ? s.iters : 0;
        return res;
    }
    return riemann_root_finish<N>(k, s);
}

// u* and the sampled state of a converged (or given-up) solve.
template <int N>
__device__ inline RiemannResult riemann_root_finish(const RiemannConsts &k, const RootSolve &s) {
    RiemannResult res;
    const RiemannSide &A = s.A, &B = s.B;
    const bool mir = s.mir;
    double fAs = s.fAs, fBs = s.fBs, qAs = s.qAs, qBs = s.qBs;
    const double p = s.p;
    const double pstar = p;
    res.pstar = pstar;
    if (s.iters < 0) {
        double invp = frcp(pstar), fdA, fdB, qA, qB;
        bool rA, rB;
        pressure_fn_root<N>(A, pstar, invp, fAs, fdA, qA, rA);
        pressure_fn_root<N>(B, pstar, invp, fBs, fdB, qB, rB);
        qAs = rA ? qA : -1.;
        qBs = rB ? qB : -1.;
    }
    res.iters = s.iters;
    // u* of the given problem (the sorted one's, negated when mirrored)
    // .5 (uA + uB) + .5 (fB - fA) = .5 ((uA + uB) + (fB - fA)): halving is
    // exact, so one rounding of the sum, halved on the integer pipe
    const double ustar = flip_if(half_of(addr(addr(A.u, B.u), subr(fBs, fAs))), mir);
    // --- sampling at S = 0: side s of the contact, as the left side
    const bool right = dneg(ustar);               // u* < 0: the right state
    const bool useB = right != mir;               // where side s sits in the sorted problem
    const double rho_s = useB ? B.rho : A.rho, p_s = useB ? B.p : A.p, c_s = useB ? B.c : A.c;
    const double invp_s = useB ? B.invp : A.invp, q_s = useB ? qBs : qAs;
    // the side's velocity, mirrored for the right side: the sorted problem
    // holds it negated when mirrored, so the two flips combine into useB
    const double u_s = flip_if(useB ? B.u : A.u, useB);
    const double ustar_s = flip_if(ustar, right);
    double rho, u, pp;
    if (nn_le(pstar, p_s)) {                      // rarefaction on side s
        const double sh = __dsub_rn(u_s, c_s);    // head speed
        if (!dneg(sh)) { rho = rho_s; u = u_s; pp = p_s; }
        else {
            const double q = !dneg(q_s) ? q_s : root<N>(xmul(pstar, invp_s));
            const double st = __fma_rn(-c_s, q, ustar_s);   // tail speed
            // tail < 0 puts S = 0 in the star region (left side); the right
            // side's test, tail >= 0 there, reads tail <= 0 mirrored
            const long long kst = ord_key(st);
            if (right ? kst <= 0 : kst < 0) {
                const double q2 = xmul(q, q), q3 = xmul(q2, q);
                rho = xmul(rho_s, N == 5 ? q3 : xmul(q3, q2));   // q^(N-2)
                u = ustar_s; pp = pstar;
            } else {
                const double cf = mulr(k.g5, __fma_rn(k.g7, u_s, c_s));
                double rm2;
                const double rn = pow_n<N>(mulr(cf, frcp(c_s)), rm2);
                u = cf; rho = mulr(rho_s, rm2); pp = mulr(p_s, rn);
            }
        }
    } else {                                      // shock on side s
        const double pm = xmul(pstar, invp_s);
        const double sl = __fma_rn(-c_s, fsqrt_rn(fma(k.g2, pm, k.g1)), u_s);   // shock speed
        // NaN: p_s < 0 (a reconstructed pressure of cold gas), the side's state
        if (!below_zero(sl)) { rho = rho_s; u = u_s; pp = p_s; }
        else { rho = xmul(rho_s, xmul(addr(pm, k.g6), frcp(fma(pm, k.g6, 1.)))); u = ustar_s; pp = pstar; }
    }
    res.flag = right ? 1 : -1;
    res.rho = rho; res.u = flip_if(u, right); res.p = pp;
    return res;
}

}  // namespace mlh
