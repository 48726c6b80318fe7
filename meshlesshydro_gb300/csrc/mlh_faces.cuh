// The face kernels: effective faces, states, exact Riemann solve and fluxes of
// every canonical face, and the batch of independent Riemann problems.  Each
// solver (mlh_faces0.cu, mlh_faces5.cu, mlh_faces7.cu) is a translation unit of
// its own, so that they compile in parallel.
#pragma once
#include "mlh_device.cuh"
#include "mlh_riemann.cuh"
#include "mlh_kernels.h"
#include "mlh_mlp.cuh"

namespace mlh {

// ------------------------------------------------------------------ faces

// Particles::pairwiseLimiter, Particles.cpp:1735-1785, for one side: phi0
// the reconstructed value, phi_i this side's particle value, phi_ij the value
// interpolated to the face, ad = |phi_i - phi_j|, delta1/delta2 = PSI_1/PSI_2
// ad, and i_lt_j = phi_i < phi_j (the two values differ).  Every comparison
// on integer keys (ord_key), off the FP64 pipe.  The shifts phi +- delta are
// fused multiply-adds fma(+-PSI, ad, phi): for the reference's PSI_1 = 0.5
// and PSI_2 = 0.25 the product is exact, so this is the reference's product
// then sum bit for bit, one FP64 instruction instead of two (other PSI: one
// rounding fewer).
__device__ __forceinline__ double pairwise_side(double phi0, double phi_i, double phi_ij, double ad, double psi1,
                                                double psi2, bool i_lt_j, int int_abs) {
    // the bound that is used is phi_minus = phi_min - delta1 when phi_i <
    // phi_j and phi_plus = phi_max + delta1 otherwise, and in both cases the
    // extreme it starts from is phi_i; the reference takes the shift when it
    // keeps the sign, (a >= 0 && b >= 0) || (a < 0 && b < 0), else
    // phi / (1 + delta1 / |phi|)
    // (phi / (1 + delta1 / |phi|) evaluated as phi |phi| / (|phi| + delta1),
    // one division by the Newton-Raphson reciprocal, and only where the
    // shift would change the sign; the same value to a few ulp, also for
    // |phi| = 0 and the int abs binding)
    const double shifted = fma(flip_if(psi1, i_lt_j), ad, phi_i);
    double bound = shifted;
    if ((ord_key(shifted) >= 0) != (ord_key(phi_i) >= 0)) {
        const double ra = ref_abs(phi_i, int_abs);
        bound = mulr(mulr(phi_i, ra), frcp(fma(psi1, ad, ra)));
    }
    const double t = fma(flip_if(psi2, !i_lt_j), ad, phi_ij);
    if (i_lt_j) {
        const double minPhiD2 = dlt(t, phi0) ? t : phi0;
        return dlt(minPhiD2, bound) ? bound : minPhiD2;
    }
    const double maxPhiD2 = dlt(phi0, t) ? t : phi0;
    return dlt(bound, maxPhiD2) ? bound : maxPhiD2;
}

// The pairwise limiter on both sides of a face: phi0R/phi0L the
// reconstructed values (replaced by the limited ones), phiR/phiL the values
// of particles i and j, rR/rL = |x_ij - x_i| / |x_j - x_i| and
// |x_ij - x_j| / |x_j - x_i|.  The j side's phi_i - phi_j is the exact
// negation of the i side's, so |phi_i - phi_j| is the same double on both
// sides and is computed once; phi_ij on the j side, phi_j + rL (phi_i -
// phi_j), is fma(rL, d, phi_j) with d = phi_i - phi_j.  Equal particle values
// (neither phi_i < phi_j nor phi_i > phi_j) give the particle values back.
template <bool MIDPOINT>
__device__ __forceinline__ void pairwise_limiter(const Params &p, double &phi0R, double &phi0L, double phiR,
                                                 double phiL, double rR, double rL) {
    const long long kR = ord_key(phiR), kL = ord_key(phiL);
    if (kR == kL) { phi0R = phiR; phi0L = phiL; return; }
    const bool r_lt_l = kR < kL;
    const double d = subr(phiR, phiL);
    const double ad = ref_abs(d, p.int_abs);
    // phi_ij on the two sides, phi_R + rR (phi_L - phi_R) and phi_L + rL (phi_R -
    // phi_L): with rR = rL = 1/2 both are the mean, evaluated once
    const double fR = fma(rR, -d, phiR);
    const double fL = MIDPOINT ? fR : fma(rL, d, phiL);
    phi0R = pairwise_side(phi0R, phiR, fR, ad, p.psi1, p.psi2, r_lt_l, p.int_abs);
    phi0L = pairwise_side(phi0L, phiL, fL, ad, p.psi1, p.psi2, !r_lt_l, p.int_abs);
}

// Network inputs of a face, from its face-frame problem sorted as the
// root solver sorts it (riemann_root_begin): side A the one with the lower
// pressure (particle i on ties), side B the other, the mirror image negating
// both normal velocities, so that du = uB - uA is the same in both
// orientations:  log(rhoB/rhoA), du/cA, log(pB/pA) >= 0, log(cB/cA), in single
// precision (c = sqrt(gamma p / rho)).  The network predicts
// y = log(p* / p_TR), p_TR the two-rarefaction guess of the face; p* and p_TR
// are the same for both orientations.  p_TR is exact when both waves are rarefactions and its error grows
// with the shock strength p_TR / min(pL, pR) - 1 (about 1e-6 at 0.2, 3e-3 at
// 2-4, 2e-2 beyond 4, measured on random states), so only faces with
// p_TR > PSTAR_HARD * min(pL, pR) are handed to the network; the others are
// solved from p_TR in the first pass.  Where |y| is below PSTAR_GATE the
// correction is within the network's own error (BF16 activations) and Newton
// starts from p_TR as well.
constexpr double PSTAR_HARD = 2.0;
constexpr float PSTAR_GATE = 0.01f;

__device__ __forceinline__ float4 pstar_features_sorted(double rhoA, double pA, double rhoB, double pB, double du,
                                                       float gamma) {
    const float ra = (float)rhoA, rb = (float)rhoB, pa = (float)pA, pb = (float)pB;
    const float ca = sqrtf(gamma * pa / ra), cb = sqrtf(gamma * pb / rb);
    return make_float4(logf(rb / ra), (float)du / ca, logf(pb / pa), logf(cb / ca));
}

// the same from the unsorted face-frame states (R = particle i, left; L = j)
__device__ __forceinline__ float4 pstar_features(const double *R, const double *L, double unR, double unL,
                                                double gamma) {
    const bool mir = dlt(L[1], R[1]);
    return mir ? pstar_features_sorted(L[0], L[1], R[0], R[1], unL - unR, (float)gamma)
               : pstar_features_sorted(R[0], R[1], L[0], L[1], unL - unR, (float)gamma);
}

// One canonical face (i < j): effective face A_ij = psi~_j(x_i)/omega_i -
// psi~_i(x_j)/omega_j from the psi~ of both slots (compEffectiveFace,
// Particles.cpp:1290-1311, 2504-2531); boosted, reconstructed, optionally
// pairwise-limited and half-step-predicted states (compRiemannStatesLR,
// :1488-1733 / 2533-2683, including the vz[i] of :1717,1719); the face-frame
// problem (normal velocity components, face_normal), exact solve with i as
// the left state, back to the lab frame and projection on A_ij
// (Riemann::Riemann/exact/rotateAndProjectFluxes2D/3D,
// demonstrator/src/Riemann.cpp:7-229; project_flux says why no rotation
// matrix is needed).  Output slot order: [mass, energy, px, py, pz].
// MODE 0: the whole face.  MODE 1 (learned guess, first pass): faces with a
// strong shock in p_TR stop before the exact solve and are
// queued (state and network inputs at the queue position, order immaterial:
// each face writes only its own flux); all other faces are finished as in
// MODE 0.  MODE 2 (second pass, over the queue): reload the state, solve from
// the network's guess, project the flux.  `harvest` (MODE 0) records network
// inputs and targets log(p*/p_TR) of every `stride`-th face.
// MODE 3 (plain first pass, root solver): one Newton step from the
// two-rarefaction guess; faces that have not converged are queued with their
// iterate, so that the warps of this pass do not all run the second step that
// a fifth of the faces need (nearly every warp holds one).  MODE 4 (second
// pass over that queue): continue Newton from the stored iterate, which is the
// same iteration with the same arithmetic, densely packed.  A full queue
// keeps the face in MODE 3 and finishes it there.
// Riemann::Riemann (demonstrator/src/Riemann.cpp:7-81) rotates both states
// with Helper::rotationMatrix2D/3D(hatA, unitX) (Helper.cpp:39-77), hatA =
// A/|A|.  The one-dimensional problem reads only the first rotated velocity
// component, and the first row of that rotation is hatA: u = hatA . v.  The
// velocities themselves stay unrotated (see project_flux).
struct FaceNormal {
    double AA, iAN;     // |A|^2, 1 / |A|
    double unR, unL;    // their velocity components along the normal A / |A|
};
template <int D>
__device__ __forceinline__ FaceNormal face_normal(const double *A, const double *R, const double *L) {
    FaceNormal fn;
    fn.AA = dotD<D>(A, A);
    fn.iAN = frsqrt(fn.AA);
    fn.unR = mulr(fn.iAN, dotD<D>(A, R + 2));
    fn.unL = mulr(fn.iAN, dotD<D>(A, L + 2));
    return fn;
}

// Riemann::exact after the solve and rotateAndProjectFluxes2D/3D
// (demonstrator/src/Riemann.cpp:100-229): the sampled velocity takes its
// tangential components from the sampled side, is rotated back and boosted by
// the frame velocity, and the flux is projected on A_ij.  Rotating a state
// into the face frame, replacing its normal component by u* and rotating back
// leaves its tangential part unchanged, so v* = v_side + (u* - u_side) hatA,
// without the rotation matrices.  R (particle i, the
// left state) and L: [rho, P, v..] with unrotated velocities, unR/unL their
// normal components.  Fo: [mass, energy, px, py, pz].  Returns ST_VACUUM
// when the solution is vacuum, else 0.
template <int D>
__device__ __forceinline__ unsigned project_flux(const RiemannResult &rs, const double *R, const double *L,
                                                 const FaceNormal &fn, const double *A, const double *vf,
                                                 double inv_gm1, int mfm, double *Fo) {
    unsigned st = 0;
    double vSol[3] = {0., 0., 0.};
    // v* = v_side + s A with s = (u* - u_side) / |A|, and A . v* = u* |A|; for
    // vacuum v_side = 0 and u* = 0
    const bool left = rs.flag == 1, vacuum = rs.flag != 1 && rs.flag != -1;
    if (vacuum) st = ST_VACUUM;
    const double sA = mulr(subr(rs.u, vacuum ? 0. : left ? fn.unL : fn.unR), fn.iAN);
#pragma unroll
    for (int a = 0; a < D; ++a) vSol[a] = fma(sA, A[a], vacuum ? 0. : left ? L[2 + a] : R[2 + a]);
    // F_m = rho* (A . v*), F_p = F_m v_lab + P* A,
    // F_E = (A . v*) (P*/(gamma-1) + rho*/2 |v_lab|^2) + P* (A . v_lab);
    // MESHLESS_FINITE_MASS keeps F_m and drops the advective terms
    const double rhoSol = rs.rho, PSol = rs.p;
    const double pe = xmul(PSol, inv_gm1);
    const double Av = mulr(rs.u, mulr(fn.AA, fn.iAN));
    double vLab[3] = {0., 0., 0.};
#pragma unroll
    for (int a = 0; a < D; ++a) vLab[a] = addr(vSol[a], vf[a]);
    Fo[0] = mulr(rhoSol, Av);
    const double Avm = mfm ? 0. : Av;
    const double mflux = mfm ? 0. : Fo[0];
#pragma unroll
    for (int a = 0; a < D; ++a) Fo[2 + a] = fma(mflux, vLab[a], mulr(PSol, A[a]));
    if (D == 2) Fo[4] = 0.;
    // pe + rho*/2 |v_lab|^2 as one fused multiply-add
    Fo[1] = fma(Avm, fma(half_of(rhoSol), dotD<D>(vLab, vLab), pe), mulr(PSol, dotD<D>(A, vLab)));
    return st;
}

// Register caps of the face kernels (MLH_FACE_MAXREG_*): with the roots and products on the integer
// pipe the passes wait on latency at 16 warps per SM.  k_faces_block: 80, three
// blocks of 256 threads (24 warps) per SM.  With 128 threads the pass over the Sedov
// 128^3 faces at 104 / 96 / 88 / 80 / 72 registers took 13.84 / 13.30 / 13.33 / 13.25 /
// 13.41 ms, that over those of 64 KH members at 80 / 72 / 64 2.65 / 2.63 / 2.74 ms; with
// 256 threads 12.47 at 80, 13.63 at 84 (two blocks), 2.52 and 2.47 ms (KH) at 72 and
// 80.  k_faces in 2D: 72.  The grid is a multiple of the blocks that reside at once
// (face_blocks): 8 blocks per SM at 96 registers left the second of two rounds
// 3/5 full, 16.4 ms.  What the pass does per face: 192 FP64 operations among 5400
// instructions, more than the instruction cache holds (no-instruction stalls a
// sixth of the time at 128 threads); a block's warps run in step between its
// barriers and share what is fetched.
#define MLH_FACE_BOUNDS __maxnreg__(D == 3 ? MLH_FACE_MAXREG_3D : MLH_FACE_MAXREG_2D)
// The face-frame Riemann problem of canonical face f (i < j): effective face
// A_ij = psi~_j(x_i)/omega_i - psi~_i(x_j)/omega_j from the psi~ of both
// slots (compEffectiveFace, Particles.cpp:1290-1311, 2504-2531); boosted,
// reconstructed, optionally pairwise-limited and half-step-predicted states
// (compRiemannStatesLR, :1488-1733 / 2533-2683, including the vz[i] of
// :1717,1719); the face normal and the normal velocity components
// (face_normal).  MID: the first-order quadrature point, the midpoint of x_i and
// x_j (else x_i + h/4 (x_j - x_i)).  It is a parameter of the kernel, not a test:
// the other point's few FP64 instructions under a test were issued with their
// lanes off, which holds the FP64 pipe as long (27 of 260 warp instructions per
// 32 faces in 3D), and out of line they cost registers.  R (particle i, the left state) and L: [rho, P, v..] with
// unrotated velocities.  Returns false for a face without its links (the
// status bit is set).
template <int D, bool MID>
__device__ __forceinline__ bool face_states(const Params &p, const Member *__restrict__ members,
                                            const int *__restrict__ memberOf, const GridInfo *__restrict__ grids,
                                            const Prim *__restrict__ prim, const Geo *__restrict__ geo,
                                            const Grad *__restrict__ grad, const uint32_t *__restrict__ nbr,
                                            const double *__restrict__ psi, const FaceRef *__restrict__ faces,
                                            const double *__restrict__ dtp, int f, unsigned &st_local, double *R,
                                            double *L, double *A, double *vf, FaceNormal &fn) {
    constexpr int NV = D + 2;
    const FaceRef fr = faces[f];
    if (fr.i < 0 || fr.slot < 0) {
        st_local |= ST_ASYMMETRIC;
        return false;
    }
    const int i = fr.i;
    const int mi = memberOf ? memberOf[i] : 0;
    const double dt = dtp[mi];
    const size_t si = (size_t)i * p.K + fr.slot;
    const uint32_t e = nbr[si];
    const int j = (int)(e & IDX_MASK);
    const bool img = (e >> IMG_SHIFT) != 0;
    const Prim pi = prim[i], pj = prim[j];
    double xi[3] = {pi.x, pi.y, pi.z}, xj[3];
    if (img) neighbour_pos<D>(e, pj, grids[mi], xj);
    else { xj[0] = pj.x; xj[1] = pj.y; xj[2] = pj.z; }
    // --- states at the face
    double xijxi[3], xjxi[3], xijxj[3];
    const double hq = MID ? 0. : p.adaptive_h ? p.hp[i] : members[mi].h;   // quadrature-point radius
#pragma unroll
    for (int a = 0; a < D; ++a) {
        xjxi[a] = subr(xj[a], xi[a]);
        if (MID) {
            // .5 (x_j - x_i) (on the integer pipe), and .5 (x_i - x_j) is its
            // exact negation
            xijxi[a] = half_of(xjxi[a]);
            xijxj[a] = flip_if(xijxi[a], true);
        } else {
            const double xij = fma(hq / 4., xjxi[a], xi[a]);
            xijxi[a] = subr(xij, xi[a]);
            xijxj[a] = subr(xij, xj[a]);
        }
    }
    const double vi[3] = {pi.vx, pi.vy, pi.vz}, vj[3] = {pj.vx, pj.vy, pj.vz};
    // v_i - v_f and v_j - v_f; with the midpoint the frame moves with the mean, and
    // they are (v_i - v_j) / 2 and its exact negation
    double wi[3] = {0., 0., 0.}, wj[3] = {0., 0., 0.};
    if (MID) {
#pragma unroll
        for (int a = 0; a < D; ++a) {
            const double mean = half_of(addr(vi[a], vj[a])), half = half_of(subr(vi[a], vj[a]));
            vf[a] = p.move ? mean : 0.;
            wi[a] = p.move ? half : vi[a];
            wj[a] = p.move ? flip_if(half, true) : vj[a];
        }
    } else {
        if (p.move) {
            const double dotProd = dotD<D>(xijxi, xjxi);
            const double dSqr = dotD<D>(xjxi, xjxi);
#pragma unroll
            for (int a = 0; a < D; ++a) vf[a] = addr(vi[a], mulr(subr(vj[a], vi[a]), dotProd) / dSqr);
        }
#pragma unroll
        for (int a = 0; a < D; ++a) { wi[a] = subr(vi[a], vf[a]); wj[a] = subr(vj[a], vf[a]); }
    }
    const double *Gi = grad[i].g, *Gj = grad[j].g;
    // gradient blocks: 0 rho, 3 vx, 6 vy, 9 vz, 12 P
    R[0] = pi.rho; L[0] = pj.rho;
    R[1] = pi.P; L[1] = pj.P;
#pragma unroll
    for (int a = 0; a < D; ++a) { R[2 + a] = wi[a]; L[2 + a] = wj[a]; }
    // W -= dt/2 (source + (v - v_frame) . grad W): the sources come with the
    // gradients (Grad::t).  The reference uses vz[i] on the j side of the vx and
    // vy terms in 3D (Particles.cpp:1717,1719).
    const double nhdt = flip_if(half_of(dt), true);
    const double *Ti = grad[i].t, *Tj = grad[j].t;
    const int blk[5] = {0, 12, 3, 6, 9};   // gradient blocks: 0 rho, 3 vx, 6 vy, 9 vz, 12 P
    if (D == 2 && !p.pairwise) {
        // no limiter between reconstruction and prediction: one FMA chain per
        // field and side, W - dt/2 source + grad W . (x_ij - x_side - dt/2 (v - v_frame))
        // (a run-wide branch: with the limiter on, image faces that skip it
        // keep the other form, so that warps do not run both; 3D keeps the
        // other form, whose registers the 3D face kernels are tuned to)
        double yi[3], yj[3];
#pragma unroll
        for (int a = 0; a < D; ++a) {
            yi[a] = fma(nhdt, wi[a], xijxi[a]);
            yj[a] = MID ? flip_if(yi[a], true) : fma(nhdt, wj[a], xijxj[a]);
        }
        if (MID && !p.move) {   // both sides advected with their own velocity
#pragma unroll
            for (int a = 0; a < D; ++a) yj[a] = fma(nhdt, wj[a], xijxj[a]);
        }
#pragma unroll
        for (int f = 0; f < NV; ++f) {
            R[f] = fma_dotD<D>(Gi + blk[f], yi, fma(nhdt, Ti[f], R[f]));
            L[f] = fma_dotD<D>(Gj + blk[f], yj, fma(nhdt, Tj[f], L[f]));
        }
    } else {
        // image faces skip the limiter (Particles.cpp:2533-2683)
        const bool limit = p.pairwise && (!img || p.img_pw);
        // |x_ij - x_i| / |x_j - x_i| and |x_ij - x_j| / |x_j - x_i|: with the
        // first-order quadrature point x_ij - x_i = (x_j - x_i) / 2 exactly,
        // so both quotients are exactly 0.5
        double ri = .5, rj = .5;
        if (!MID && limit) {
            double xijxi_abs = 0., xijxj_abs = 0., xjxi_abs = 0.;
#pragma unroll
            for (int a = 0; a < D; ++a) {
                xijxi_abs = fma(xijxi[a], xijxi[a], xijxi_abs);
                xijxj_abs = fma(xijxj[a], xijxj[a], xijxj_abs);
                xjxi_abs = fma(xjxi[a], xjxi[a], xjxi_abs);
            }
            xjxi_abs = sqrt(xjxi_abs);
            ri = sqrt(xijxi_abs) / xjxi_abs;
            rj = sqrt(xijxj_abs) / xjxi_abs;
        }
        const double wq[3] = {wj[0], wj[1], wi[2]};
        // field by field, so that one field's gradients and particle values are
        // live at a time: W + grad W . (x_ij - x_side), one FMA chain from W; the
        // limiter; the prediction, one FMA chain per side from the limited value
#pragma unroll
        for (int f = 0; f < NV; ++f) {
            double r = fma_dotD<D>(Gi + blk[f], xijxi, R[f]), l = fma_dotD<D>(Gj + blk[f], xijxj, L[f]);
            if (limit) pairwise_limiter<MID>(p, r, l, R[f], L[f], ri, rj);
            R[f] = fma(nhdt, fma_dotD<D>(wi, Gi + blk[f], Ti[f]), r);
            L[f] = fma(nhdt, fma_dotD<D>((D == 3 && (f == 2 || f == 3)) ? wq : wj, Gj + blk[f], Tj[f]), l);
        }
    }
    if (dneg(R[1]) || dneg(L[1])) st_local |= ST_NEG_PRESSURE;
    // --- effective face, from V_i psi~_j(x_i) of both slots
    {
        const double *ps_i = psi + si * 3;
        if (fr.rslot >= 0) {
            const double *ps_j = psi + ((size_t)j * p.K + fr.rslot) * 3;
#pragma unroll
            for (int a = 0; a < D; ++a) A[a] = subr(ps_i[a], ps_j[a]);
        } else {
            st_local |= ST_ASYMMETRIC;
#pragma unroll
            for (int a = 0; a < D; ++a) A[a] = ps_i[a];
        }
    }
    // --- Riemann problem in the face frame (i left, j right)
    fn = face_normal<D>(A, R, L);
    return true;
}

// The faces of a thread's rounds (f0, f0 + stride, ..) that the root solver does not
// take, by riemann_exact: set up again, after the kernel's own loop, which skipped
// them, so that the powers' calls shape no register of it (in the loop they cost the
// pass 2-6 % at gamma = 7/5, also where every face is taken).
template <int D, int ROOT, bool MID>
__device__ __forceinline__ void general_faces(const Params &p, const RiemannConsts &rc, const Member *__restrict__ members,
                                              const int *__restrict__ memberOf, const GridInfo *__restrict__ grids,
                                              const Prim *__restrict__ prim, const Geo *__restrict__ geo,
                                              const Grad *__restrict__ grad, const uint32_t *__restrict__ nbr,
                                              const double *__restrict__ psi, const FaceRef *__restrict__ faces,
                                              const double *__restrict__ dtp, double *__restrict__ Fface, int f0, int nf,
                                              int stride, unsigned &st_local, unsigned long long &iters_local) {
    for (int f = f0; f < nf; f += stride) {
        double R[5], L[5], A[3] = {0., 0., 0.}, vf[3] = {0., 0., 0.};
        FaceNormal fn = {};
        if (!face_states<D, MID>(p, members, memberOf, grids, prim, geo, grad, nbr, psi, faces, dtp, f, st_local, R, L, A,
                                 vf, fn) ||
            root_takes<ROOT>(R[0], fn.unR, R[1], L[0], fn.unL, L[1]))
            continue;
        const RiemannResult rs = riemann_exact(rc, R[0], fn.unR, R[1], L[0], fn.unL, L[1]);
        if (rs.iters < 0) st_local |= ST_NEWTON;
        else iters_local += (unsigned long long)rs.iters;
        double Fo[5];
        st_local |= project_flux<D>(rs, R, L, fn, A, vf, rc.inv_gm1, p.mfm, Fo);
        double2 *dst = reinterpret_cast<double2 *>(Fface + (size_t)f * 6);
        dst[0] = make_double2(Fo[0], Fo[1]);
        dst[1] = make_double2(Fo[2], Fo[3]);
        dst[2] = make_double2(Fo[4], (double)rs.iters);
    }
}

template <int D, int ROOT, int MODE, bool MID>
__global__ void MLH_FACE_BOUNDS k_faces(Params p, RiemannConsts rc, const Member *__restrict__ members,
                                               const int *__restrict__ memberOf, const GridInfo *__restrict__ grids,
                                               const Prim *__restrict__ prim, const Geo *__restrict__ geo,
                                               const Grad *__restrict__ grad, const uint32_t *__restrict__ nbr,
                                               const double *__restrict__ psi, const int *__restrict__ faceTotal,
                                               const FaceRef *__restrict__ faces, const double *__restrict__ dtp,
                                               double *__restrict__ Fface, unsigned long long *__restrict__ newtonSum,
                                               unsigned *__restrict__ status, FaceQueue qa, FaceQueue qb,
                                               float4 *__restrict__ feat, const float *__restrict__ yguess,
                                               Harvest hv) {
    if (step_aborted(status)) return;   // no valid faces
    int nf = *faceTotal < p.faces_cap ? *faceTotal : p.faces_cap;
    constexpr bool QUEUED = MODE == 2 || MODE == 4;   // passes over the queue
    constexpr bool SOME = ROOT == 7 && !QUEUED;       // the solver does not take every face
    bool general = false;
    if (QUEUED) {   // the queue holds min(count, capacity) faces; MODE 3 finished the rest itself
        const int qn = *qa.count < qa.cap ? *qa.count : qa.cap;
        nf = qn < nf ? qn : nf;
    }
    const double gamma = p.gamma;
    unsigned long long iters_local = 0, fallback_local = 0, deferred_local = 0;
    unsigned st_local = 0;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < nf; t += gridDim.x * blockDim.x) {
        // MODE 2 walks the queue: t is the queue position, f the face
        const int f = QUEUED ? qa.face[t] : t;
        double R[5], L[5], A[3] = {0., 0., 0.}, vf[3] = {0., 0., 0.};
        FaceNormal fn = {};
        double ptr_q = -1.;   // MODE 2: two-rarefaction guess found in MODE 1; MODE 4: Newton iterate
        if (QUEUED) {
            const FaceState &fs = qa.st[t];
            ptr_q = fs.v[16];
#pragma unroll
            for (int k = 0; k < 5; ++k) { R[k] = fs.v[k]; L[k] = fs.v[5 + k]; }
#pragma unroll
            for (int a = 0; a < 3; ++a) { A[a] = fs.v[10 + a]; vf[a] = fs.v[13 + a]; }
            fn = face_normal<D>(A, R, L);
        } else {
        if (!face_states<D, MID>(p, members, memberOf, grids, prim, geo, grad, nbr, psi, faces, dtp, f, st_local, R, L, A,
                            vf, fn))
            continue;
        if (SOME && !root_takes<ROOT ? ROOT : 5>(R[0], fn.unR, R[1], L[0], fn.unL, L[1])) { general = true; continue; }
        }   // !QUEUED
        const double unR = fn.unR, unL = fn.unL;
        double guess = -1.;
        if (MODE == 2) {
            const float y = yguess[t];
            if (isfinite(y) && fabsf(y) > PSTAR_GATE && fabsf(y) < 30.f)
                guess = ptr_q * (double)__expf(y);
        }
        if (MODE == 4) guess = ptr_q;
        // MODE 1 defers faces whose two-rarefaction guess says strong shock
        const double defer = MODE == 1 ? PSTAR_HARD * (dlt(L[1], R[1]) ? L[1] : R[1]) : 0.;   // min on the keys
        RiemannResult rs = ROOT ? riemann_exact_root<ROOT ? ROOT : 5>(rc, R[0], unR, R[1], L[0], unL, L[1], guess, defer,
                                                  (MODE == 3 || (MODE == 1 && p.face_split)) ? 1 : 0)
                                 : riemann_exact(rc, R[0], unR, R[1], L[0], unL, L[1], guess, defer);
        // deferred faces: strong shocks of MODE 1 (unsolved, iters 0) go to
        // queue A for the network; faces Newton has not finished after one
        // step go to queue A (MODE 3) or B (MODE 1) with their iterate
        if ((MODE == 1 || MODE == 3) && rs.flag == 2) {
            const bool strong = MODE == 1 && rs.iters == 0;
            const FaceQueue &fq = (MODE == 1 && !strong) ? qb : qa;
            const int q = atomicAdd(fq.count, 1);
            if (q < fq.cap) {
                FaceState &fs = fq.st[q];
#pragma unroll
                for (int k = 0; k < 5; ++k) { fs.v[k] = R[k]; fs.v[5 + k] = L[k]; }
#pragma unroll
                for (int a = 0; a < 3; ++a) { fs.v[10 + a] = A[a]; fs.v[13 + a] = vf[a]; }
                fs.v[16] = rs.pstar;   // the two-rarefaction guess (strong) or the Newton iterate
                fq.face[q] = f;
                if (strong) feat[q] = pstar_features(R, L, unR, unL, gamma);
                else iters_local += (unsigned long long)rs.iters;
                continue;
            }
            // queue full: finish here, from the iterate or from p_TR
            const int done = rs.iters;
            rs = ROOT ? riemann_exact_root<ROOT ? ROOT : 5>(rc, R[0], unR, R[1], L[0], unL, L[1], strong ? -1. : rs.pstar, 0.)
                       : riemann_exact(rc, R[0], unR, R[1], L[0], unL, L[1], -1., 0.);
            if (rs.iters >= 0) rs.iters += done;
        }
        if (MODE == 0 && hv.stride > 0 && (hv.strong || f % hv.stride == 0)) {
            const double ptr = two_rarefaction_guess<ROOT>(rc, R[0], unR, R[1], L[0], unL, L[1]);
            if (rs.iters >= 0 && rs.pstar > 0. && ptr > 0.) {
                if (hv.strong) {
                    // the faces the learned step hands to the network
                    if (dlt(PSTAR_HARD * (dlt(L[1], R[1]) ? L[1] : R[1]), ptr)) {
                        const int slot = atomicAdd(hv.count, 1);
                        if (slot < hv.cap) {
                            hv.x[slot] = pstar_features(R, L, unR, unL, gamma);
                            hv.t[slot] = (float)log(rs.pstar / ptr);
                        }
                    }
                } else {
                    const int slot = f / hv.stride;
                    if (slot < hv.cap) {
                        hv.x[slot] = pstar_features(R, L, unR, unL, gamma);
                        hv.t[slot] = (float)log(rs.pstar / ptr);
                        atomicMax(hv.count, slot + 1);
                    }
                }
            }
        }
        if (rs.iters < 0) st_local |= ST_NEWTON;
        else {
            // iters counts every Newton step run: a learned guess that did not
            // converge adds max_iter wasted steps before the restart from the
            // two-rarefaction guess
            if (MODE == 2 && rs.iters > rc.max_iter) ++fallback_local;
            if (MODE == 2) ++deferred_local;
            iters_local += (unsigned long long)rs.iters;
        }
        double Fo[5];
        st_local |= project_flux<D>(rs, R, L, fn, A, vf, rc.inv_gm1, p.mfm, Fo);
        // the face's Newton steps (the step of the first pass included in
        // MODE 4; -1: no convergence) in the record's sixth double, for parity
        // checks
        const int face_iters = rs.iters < 0 ? -1 : rs.iters + (MODE == 4 ? 1 : 0);
        double2 *dst = reinterpret_cast<double2 *>(Fface + (size_t)f * 6);
        dst[0] = make_double2(Fo[0], Fo[1]);
        dst[1] = make_double2(Fo[2], Fo[3]);
        dst[2] = make_double2(Fo[4], (double)face_iters);
    }
    if (SOME && general)
        general_faces<D, ROOT ? ROOT : 5, MID>(p, rc, members, memberOf, grids, prim, geo, grad, nbr, psi, faces, dtp, Fface,
                                               blockIdx.x * blockDim.x + threadIdx.x, nf, gridDim.x * blockDim.x, st_local,
                                               iters_local);
    // block-level accumulation of the counters
    for (int o = 16; o > 0; o >>= 1) {
        iters_local += __shfl_xor_sync(0xffffffffu, iters_local, o);
        fallback_local += __shfl_xor_sync(0xffffffffu, fallback_local, o);
        deferred_local += __shfl_xor_sync(0xffffffffu, deferred_local, o);
        st_local |= __shfl_xor_sync(0xffffffffu, st_local, o);
    }
    if ((threadIdx.x & 31) == 0) {
        if (iters_local) atomicAdd(newtonSum, iters_local);
        if (fallback_local) atomicAdd(newtonSum + 1, fallback_local);
        if (deferred_local) atomicAdd(newtonSum + 2, deferred_local);
        if (st_local) flag(status, st_local);
    }
}

// Plain root-solver face pass with the faces that need more than one Newton
// step regrouped inside the block (face_split 2).  A warp issues every
// instruction that any of its lanes needs, so the second Newton step of the
// few faces that need it would hold the whole warp.  Instead: every face of
// the block's round sets up its problem and takes the first Newton step
// from p_TR, and leaves its solver state (sorted sides, iterate) in shared
// memory; the block's unfinished faces are listed and continued, densely, by
// its first threads (the iteration riemann_exact_root runs from the iterate as a
// guess, on the stored sides: the same arithmetic as the two-pass split);
// then every face samples its solution and projects its flux, with all
// lanes busy.  The loop runs in block-wide rounds so that every thread
// reaches the barriers.  LEARNED: the learned-guess step.  Strong shocks
// (p_TR > PSTAR_HARD min(pL, pR)) stop before their first Newton step; the
// block lists them, evaluates the network for them on the tensor cores (a
// warp per 16 faces, block_network_guess; a block-uniform branch that a round
// without strong shocks skips) and continues them from p_TR e^y together with
// the other unfinished faces.  Nothing leaves the block: the plain and the
// learned step differ only by that branch.

// The network's guesses for the ns strong-shock faces of a round listed in
// slist (their solver states in sv, s.p = p_TR): warp w takes the faces
// w*16 .. w*16+15, then the next FB_T / 2, and so on; s.p becomes p_TR e^y where
// PSTAR_GATE < |y| < 30 (finite), and stays p_TR elsewhere.  Every lane of a
// warp runs the MMAs (rows beyond ns are zero inputs whose outputs are
// dropped).  Out of line, so that the rare branch that calls it does not shape
// the register allocation of the face pass.
static __device__ __noinline__ void block_network_guess(const PackedMlp *__restrict__ w, RootSolve *sv, const int *slist,
                                                 int ns, float gamma) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int base = warp * 16; base < ns; base += FB_T / 2) {
        const int row = base + (lane & 15);
        const bool mine = lane < 16 && row < ns;
        float4 xi = make_float4(0.f, 0.f, 0.f, 0.f);
        if (mine) {
            const RootSolve &q = sv[slist[row]];
            xi = pstar_features_sorted(q.A.rho, q.A.p, q.B.rho, q.B.p, q.du, gamma);
        }
        const float y = mlp_rows<1>(w, xi);
        if (mine && isfinite(y) && fabsf(y) > PSTAR_GATE && fabsf(y) < 30.f) {
            RootSolve &q = sv[slist[row]];
            q.p = q.p * (double)__expf(y);
        }
    }
}

template <int D, int ROOT, bool LEARNED>
__global__ void __maxnreg__(MLH_FACE_MAXREG_BLOCK) k_faces_block(Params p, RiemannConsts rc, const Member *__restrict__ members,
                                              const int *__restrict__ memberOf, const GridInfo *__restrict__ grids,
                                              const Prim *__restrict__ prim, const Geo *__restrict__ geo,
                                              const Grad *__restrict__ grad, const uint32_t *__restrict__ nbr,
                                              const double *__restrict__ psi, const int *__restrict__ faceTotal,
                                              const FaceRef *__restrict__ faces, const double *__restrict__ dtp,
                                              double *__restrict__ Fface, unsigned long long *__restrict__ newtonSum,
                                              unsigned *__restrict__ status, const PackedMlp *__restrict__ mlp,
                                              int *__restrict__ generalCount) {
    __shared__ RootSolve sv[FB_T];
    __shared__ int todo[FB_T];
    __shared__ int slist[LEARNED ? FB_T : 1];
    __shared__ int wcount[FB_T / 32];
    if (step_aborted(status)) return;   // no valid faces
    const int nf = *faceTotal < p.faces_cap ? *faceTotal : p.faces_cap;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned long long iters_local = 0, fallback_local = 0, learned_local = 0;
    unsigned st_local = 0;
    for (int t0 = blockIdx.x * FB_T; t0 < nf; t0 += gridDim.x * FB_T) {
        const int f = t0 + threadIdx.x;
        double R[5], L[5], A[3] = {0., 0., 0.}, vf[3] = {0., 0., 0.};
        FaceNormal fn = {};
        bool valid = f < nf;
        if (valid)
            valid = face_states<D, true>(p, members, memberOf, grids, prim, geo, grad, nbr, psi, faces, dtp, f, st_local, R,
                                   L, A, vf, fn);
        if (ROOT == 7 && valid && !root_takes<ROOT>(R[0], fn.unR, R[1], L[0], fn.unL, L[1])) {
            *generalCount = 1;   // left to k_faces_general
            valid = false;
        }
        bool unfinished = false, strong = false;
        if (valid) {
            // strong shocks of the learned step stop before their first
            // Newton step: p_TR > PSTAR_HARD min(pL, pR) (min on the keys)
            const double defer = LEARNED ? PSTAR_HARD * (dlt(L[1], R[1]) ? L[1] : R[1]) : 0.;
            const RootSolve s0 = riemann_root_begin<ROOT>(rc, R[0], fn.unR, R[1], L[0], fn.unL, L[1], -1., defer, 1);
            sv[threadIdx.x] = s0;
            unfinished = s0.stage == 2;
            strong = LEARNED && s0.stage == 3;
        }
        // --- list the block's unfinished faces (and, learned, its strong shocks)
        const unsigned bal = __ballot_sync(0xffffffffu, unfinished || strong);
        const unsigned sbal = LEARNED ? __ballot_sync(0xffffffffu, strong) : 0u;
        if (lane == 0) wcount[warp] = __popc(bal) | (__popc(sbal) << 16);
        __syncthreads();
        int before = 0, nu = 0, sbefore = 0, ns = 0;
#pragma unroll
        for (int w = 0; w < FB_T / 32; ++w) {
            const int c = wcount[w] & 0xffff, cs = wcount[w] >> 16;
            before += w < warp ? c : 0;
            nu += c;
            sbefore += w < warp ? cs : 0;
            ns += cs;
        }
        const unsigned below = (1u << lane) - 1u;
        if (unfinished || strong) todo[before + __popc(bal & below)] = threadIdx.x;
        if (LEARNED && strong) slist[sbefore + __popc(sbal & below)] = threadIdx.x;
        __syncthreads();
        if (LEARNED && ns > 0) {   // block-uniform
            block_network_guess(mlp, sv, slist, ns, (float)p.gamma);
            __syncthreads();
        }
        // --- continue them on the first nu threads
        if ((int)threadIdx.x < nu) {
            const int slot = todo[threadIdx.x];
            RootSolve c = sv[slot];
            const bool from_net = LEARNED && c.stage == 3;
            riemann_root_continue<ROOT>(rc, c);
            if (from_net) {
                ++learned_local;
                if (c.iters > rc.max_iter) ++fallback_local;
            }
            sv[slot] = c;
        }
        __syncthreads();
        // --- sample and project, every face of the round
        if (valid) {
            const RootSolve s = sv[threadIdx.x];
            RiemannResult rs;
            if (s.stage == 0) {
                rs.rho = 0.; rs.u = 0.; rs.p = 0.; rs.pstar = 0.; rs.flag = 0; rs.iters = 0;
            } else {
                rs = riemann_root_finish<ROOT>(rc, s);
            }
            if (unfinished) iters_local += 1;   // the first step, counted as the two-pass split counts it
            if (rs.iters < 0) st_local |= ST_NEWTON;
            else iters_local += (unsigned long long)rs.iters;
            double Fo[5];
            st_local |= project_flux<D>(rs, R, L, fn, A, vf, rc.inv_gm1, p.mfm, Fo);
            const int face_iters = rs.iters < 0 ? -1 : rs.iters + (unfinished ? 1 : 0);
            double2 *dst = reinterpret_cast<double2 *>(Fface + (size_t)f * 6);
            dst[0] = make_double2(Fo[0], Fo[1]);
            dst[1] = make_double2(Fo[2], Fo[3]);
            dst[2] = make_double2(Fo[4], (double)face_iters);
        }
        __syncthreads();   // the shared state is rewritten in the next round
    }
    for (int o = 16; o > 0; o >>= 1) {
        iters_local += __shfl_xor_sync(0xffffffffu, iters_local, o);
        if (LEARNED) {
            fallback_local += __shfl_xor_sync(0xffffffffu, fallback_local, o);
            learned_local += __shfl_xor_sync(0xffffffffu, learned_local, o);
        }
        st_local |= __shfl_xor_sync(0xffffffffu, st_local, o);
    }
    if (lane == 0) {
        if (iters_local) atomicAdd(newtonSum, iters_local);
        if (LEARNED && fallback_local) atomicAdd(newtonSum + 1, fallback_local);
        if (LEARNED && learned_local) atomicAdd(newtonSum + 2, learned_local);
        if (st_local) flag(status, st_local);
    }
}

// The faces that k_faces_block left to riemann_exact, when there are any
// (generalCount).  A kernel of its own, for gamma = 7/5 alone: at the end of
// k_faces_block the same code took registers from its loop (640^2 particles: 1277 us
// without, 1343 there, 1291 so; the clear and this launch are 7 us of it).
template <int D, int ROOT>
__global__ void MLH_FACE_BOUNDS k_faces_general(Params p, RiemannConsts rc, const Member *__restrict__ members,
                                                const int *__restrict__ memberOf, const GridInfo *__restrict__ grids,
                                                const Prim *__restrict__ prim, const Geo *__restrict__ geo,
                                                const Grad *__restrict__ grad, const uint32_t *__restrict__ nbr,
                                                const double *__restrict__ psi, const int *__restrict__ faceTotal,
                                                const FaceRef *__restrict__ faces, const double *__restrict__ dtp,
                                                double *__restrict__ Fface, unsigned long long *__restrict__ newtonSum,
                                                unsigned *__restrict__ status, const int *__restrict__ generalCount) {
    if (*generalCount == 0 || step_aborted(status)) return;
    const int nf = *faceTotal < p.faces_cap ? *faceTotal : p.faces_cap;
    unsigned long long iters_local = 0;
    unsigned st_local = 0;
    general_faces<D, ROOT, true>(p, rc, members, memberOf, grids, prim, geo, grad, nbr, psi, faces, dtp, Fface,
                                 blockIdx.x * blockDim.x + threadIdx.x, nf, gridDim.x * blockDim.x, st_local, iters_local);
    if (iters_local) atomicAdd(newtonSum, iters_local);
    if (st_local) flag(status, st_local);
}

// Riemann::Riemann + Riemann::exact (demonstrator/src/Riemann.cpp:7-229) for a
// batch of independent faces: per face the left state Wi (particle i) and the
// right state Wj (neighbour j), each [rho, P, v_x, v_y(, v_z)], the frame
// velocity and A_ij; one thread per face, the same device functions as
// k_faces.  F: [mass, energy, momentum] per face; iters: Newton iterations
// (-1 when the iteration did not converge).
template <int D, int ROOT>
__global__ void __launch_bounds__(256) k_riemann_batch(int n, RiemannConsts rc, int mfm,
                                                       const double *__restrict__ Wi, const double *__restrict__ Wj,
                                                       const double *__restrict__ vFrame,
                                                       const double *__restrict__ Aij, double *__restrict__ F,
                                                       int *__restrict__ iters, unsigned *__restrict__ status) {
    constexpr int NV = D + 2;
    unsigned st = 0;
    for (int f = blockIdx.x * blockDim.x + threadIdx.x; f < n; f += gridDim.x * blockDim.x) {
        double R[5] = {0., 0., 0., 0., 0.}, L[5] = {0., 0., 0., 0., 0.};
        double A[3] = {0., 0., 0.}, vf[3] = {0., 0., 0.};
#pragma unroll
        for (int k = 0; k < NV; ++k) { R[k] = Wi[(size_t)f * NV + k]; L[k] = Wj[(size_t)f * NV + k]; }
#pragma unroll
        for (int a = 0; a < D; ++a) { A[a] = Aij[(size_t)f * D + a]; vf[a] = vFrame[(size_t)f * D + a]; }
        if (R[1] < 0. || L[1] < 0.) st |= ST_NEG_PRESSURE;
        const FaceNormal fn = face_normal<D>(A, R, L);
        const double unR = fn.unR, unL = fn.unL;
        RiemannResult rs;
        if (ROOT == 0) rs = riemann_exact(rc, R[0], unR, R[1], L[0], unL, L[1], -1., 0.);
        else if (!root_takes<ROOT ? ROOT : 5>(R[0], unR, R[1], L[0], unL, L[1]))
            rs = riemann_exact_call(rc.gamma, rc.tol, rc.max_iter, R[0], unR, R[1], L[0], unL, L[1]);
        else rs = riemann_exact_root<ROOT ? ROOT : 5>(rc, R[0], unR, R[1], L[0], unL, L[1], -1., 0.);
        if (rs.iters < 0) st |= ST_NEWTON;
        double Fo[5];
        st |= project_flux<D>(rs, R, L, fn, A, vf, rc.inv_gm1, mfm, Fo);
#pragma unroll
        for (int k = 0; k < NV; ++k) F[(size_t)f * NV + k] = Fo[k];
        if (iters) iters[f] = rs.iters;
    }
    if (st) flag(status, st);
}

// ------------------------------------------------------------------ launchers

// The face passes of a step: the structure that the tuning chose, of the solver
// for ROOT = 2 gamma / (gamma - 1) (5, 7, or 0: any gamma, one pass).
template <int D, int ROOT>
void launch_faces(StepArgs &a) {
    const Params &p = a.p;
    cudaStream_t s = a.stream;
    const int fT = a.tune.face_threads, fB = face_grid(a, 0), fBb = face_grid(a, 2);
    Params pf = p;   // the face passes see the tuned split
    const RiemannConsts rc = make_riemann_consts(p.gamma, p.rtol, p.rmaxit);
    const FaceQueue qa{a.fstate, a.queueFace, a.queueCount, a.qcap};
    const FaceQueue qb{a.fstate2, a.queueFace2, a.queueCount2, a.qcap2};
#define MLH_FACES(MODE, MID, QA, QB)                                                                              \
    k_faces<D, ROOT, MODE, MID><<<fB, fT, 0, s>>>(pf, rc, a.members, a.memberOf, a.grids, a.prim, a.geo, a.grad,  \
                                                  a.nbr, a.psi, a.faceOff + p.n, a.faces, a.dt, a.Fface,          \
                                                  a.newtonSum, a.status, QA, QB, a.feat, a.yguess, a.harvest)
#define MLH_FACES_MID(MODE, QA, QB)                     \
    do {                                                \
        if (p.foqp) MLH_FACES(MODE, true, QA, QB);      \
        else MLH_FACES(MODE, false, QA, QB);            \
    } while (0)
#define MLH_FACES_GENERAL()                                                                                       \
    do {                                                                                                          \
        if constexpr (ROOT == 7)                                                                                  \
            k_faces_general<D, ROOT><<<fB, fT, 0, s>>>(pf, rc, a.members, a.memberOf, a.grids, a.prim, a.geo,     \
                                                       a.grad, a.nbr, a.psi, a.faceOff + p.n, a.faces, a.dt,      \
                                                       a.Fface, a.newtonSum, a.status, a.queueCount);             \
    } while (0)
    // the structures that regroup unfinished faces (face_split 1, 2) are built
    // for the midpoint quadrature point; with the other one a step runs the one
    // pass (the same bits)
    const int split = p.foqp ? a.tune.face_split : 0;
    pf.face_split = split;
    if constexpr (ROOT != 0) {
        if (a.learned) {
            // strong shocks: network guess (queue A); the rest as the plain step
            cudaMemsetAsync(a.queueCount, 0, sizeof(int), s);
            if (a.queueCount2) cudaMemsetAsync(a.queueCount2, 0, sizeof(int), s);
            if (split == 2) {
                // unfinished faces continued inside the block, strong shocks from
                // the network's guess evaluated there
                k_faces_block<D, ROOT, true><<<fBb, FB_T, 0, s>>>(pf, rc, a.members, a.memberOf, a.grids, a.prim, a.geo, a.grad,
                                                           a.nbr, a.psi, a.faceOff + p.n, a.faces, a.dt, a.Fface,
                                                           a.newtonSum, a.status, (const PackedMlp *)a.mlp_packed, a.queueCount);
                MLH_FACES_GENERAL();
            } else {
                MLH_FACES_MID(1, qa, qb);
                pstar_infer_dev(a.feat, a.queueCount, (int)a.faces_cap, a.mlp_packed, a.yguess, a.sm_count, s);
                MLH_FACES(2, true, qa, qb);
                if (a.fstate2 && split == 1) MLH_FACES(4, true, qb, qb);
            }
        } else if (a.harvest.stride == 0 && split == 2) {
            // unconverged faces after one Newton step continued inside the block
            if (ROOT == 7) cudaMemsetAsync(a.queueCount, 0, sizeof(int), s);
            k_faces_block<D, ROOT, false><<<fBb, FB_T, 0, s>>>(pf, rc, a.members, a.memberOf, a.grids, a.prim, a.geo, a.grad, a.nbr,
                                                        a.psi, a.faceOff + p.n, a.faces, a.dt, a.Fface, a.newtonSum,
                                                        a.status, nullptr, a.queueCount);
            MLH_FACES_GENERAL();
        } else if (a.fstate && a.harvest.stride == 0 && split) {
            // unconverged faces after one Newton step go to a second, dense pass
            cudaMemsetAsync(a.queueCount, 0, sizeof(int), s);
            MLH_FACES(3, true, qa, qb);
            MLH_FACES(4, true, qa, qb);
        } else {
            MLH_FACES_MID(0, qa, qb);
        }
    } else {
        if (a.learned) {
            cudaMemsetAsync(a.queueCount, 0, sizeof(int), s);
            if (a.queueCount2) cudaMemsetAsync(a.queueCount2, 0, sizeof(int), s);
            MLH_FACES_MID(1, qa, qb);
            pstar_infer_dev(a.feat, a.queueCount, (int)a.faces_cap, a.mlp_packed, a.yguess, a.sm_count, s);
            MLH_FACES(2, true, qa, qb);
        } else {
            MLH_FACES_MID(0, qa, qb);
        }
    }
#undef MLH_FACES_GENERAL
#undef MLH_FACES_MID
#undef MLH_FACES
}

template <int D, int ROOT>
void launch_riemann_batch(int n, const RiemannConsts &rc, int mfm, const double *Wi, const double *Wj,
                          const double *vFrame, const double *Aij, double *F, int *iters, unsigned *status,
                          cudaStream_t s) {
    const int blocks = n > 0 ? (n + 255) / 256 : 1;
    k_riemann_batch<D, ROOT><<<blocks, 256, 0, s>>>(n, rc, mfm, Wi, Wj, vFrame, Aij, F, iters, status);
}

#define MLH_FACE_INSTANCES(ROOT)                                                                                \
    template void launch_faces<2, ROOT>(StepArgs &);                                                     \
    template void launch_faces<3, ROOT>(StepArgs &);                                                     \
    template void launch_riemann_batch<2, ROOT>(int, const RiemannConsts &, int, const double *,         \
                                                       const double *, const double *, const double *,          \
                                                       double *, int *, unsigned *, cudaStream_t);              \
    template void launch_riemann_batch<3, ROOT>(int, const RiemannConsts &, int, const double *,         \
                                                       const double *, const double *, const double *,          \
                                                       double *, int *, unsigned *, cudaStream_t);

}  // namespace mlh
