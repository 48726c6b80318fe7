// Reciprocals, roots and products of doubles on the integer pipe.
//
// GB300 runs one FP64 warp instruction per SM in 17-20 cycles and 64 issue
// slots pass meanwhile, of which the step's kernels used one in seven.  The
// functions here take a single-precision hardware estimate (MUFU) and finish
// it in 64-bit fixed point with 32 x 32 -> 64 bit multiply-adds, so that they
// occupy the FP64 pipe for nothing at all.  Measured at 12 warps per SM, SM
// cycles per warp (before -> after): reciprocal 54 -> 20, reciprocal square
// root 97 -> 29, square root 150 (sqrt) -> 36, product 20 -> 14; beside a
// stream of FP64 FMAs two reciprocals per four FMAs or one product per FMA
// cost no time that can be seen.
//
// The refinement is a series about the estimate: with y = z^(-1/N) (1 + e),
// |e| a few 2^-22, and r = 1 - z y^N,
//   z^(-1/N)    = y (1 + r/N + (1 + N) r^2 / (2 N^2) + O(r^3)),
//   z^(1 - 1/N) = z y^(N-1) (1 + a r + a (a + 1) r^2 / 2 + O(r^3)), a = (N-1)/N,
// where the dropped terms are below 2^-59, and the fixed point carries 2^-62
// or better: results are within 0.52 ulp (most are correctly rounded), against
// 0.504, 0.993 and a few ulp of the FP64 forms that they replace.
//
// Every function tests its operand's exponent field once and leaves zeros,
// subnormals, infinities, NaN and (for the roots) negative operands to the
// FP64 form, out of line, so that those have the results they always had.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace mlh {

__device__ __forceinline__ uint64_t mul_wide(uint32_t a, uint32_t b) { return (uint64_t)a * b; }
__device__ __forceinline__ uint32_t hi_word(uint64_t v) { return (uint32_t)(v >> 32); }
__device__ __forceinline__ uint64_t words(uint32_t lo, uint32_t hi) { return ((uint64_t)hi << 32) | lo; }
// floor(a u / 2^32) for signed a (below 2^63 / 2 in magnitude) and unsigned u < 2^31
__device__ __forceinline__ int64_t mul_hi32(int64_t a, uint32_t u) {
    return (int64_t)hi_word(mul_wide((uint32_t)a, u)) + (int64_t)(int32_t)(a >> 32) * (int64_t)(int32_t)u;
}

// x with its sign bit flipped when f, and |x|, on the high word alone: written
// on the 64-bit pattern or as -x and fabs, the compiler turns them into FP64
// additions wherever it cannot fold them into a consumer
__device__ __forceinline__ double flip_if(double x, bool f) {
    return __hiloint2double(__double2hiint(x) ^ ((int)f << 31), __double2loint(x));
}
__device__ __forceinline__ double abs_bits(double x) {
    return __hiloint2double(__double2hiint(x) & 0x7fffffff, __double2loint(x));
}

// a b, a + b and a - b, rounded once, as fused multiply-adds: fma(a, b, -0),
// fma(a, 1, b) and fma(b, -1, a) are the same doubles.  A DFMA whose three
// operands sit in registers holds the FP64 pipe 16.8 SM cycles per warp, a
// DADD, a DMUL or a DFMA with an immediate or a constant-bank operand 20.0
// (four chains per thread, 12 and 16 warps per SM), so the 1 and the -0 have to
// be registers that the compiler cannot see through: both are built from the
// count of SMs, whose top bit is 0.
__device__ __forceinline__ uint32_t opaque_zero() {
    uint32_t t;
    asm("mov.u32 %0, %%nsmid;" : "=r"(t));
    return t >> 31;
}
__device__ __forceinline__ double reg_one() { return __hiloint2double(0x3ff00000 + opaque_zero(), opaque_zero()); }
__device__ __forceinline__ double mulr(double a, double b) {
    return fma(a, b, __hiloint2double(0x80000000u + opaque_zero(), opaque_zero()));
}
__device__ __forceinline__ double addr(double a, double b) { return fma(a, reg_one(), b); }
__device__ __forceinline__ double subr(double a, double b) { return fma(b, -reg_one(), a); }

// FP64 forms: the hardware estimates (relative error e of a few 2^-23), each
// refined by one third-order step, 1/x = r (1 + e + e^2 + ..), e = 1 - x r,
// and 1/sqrt(x) = y (1 + e/2 + 3 e^2/8 + ..), e = 1 - x y^2.
static __device__ __noinline__ double rcp_fp64(double x) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    const double e = fma(-x, r, 1.);
    return fma(r, fma(e, e, e), r);
}
static __device__ __noinline__ double rsqrt_fp64(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-(x * y), y, 1.);
    return fma(y, e * fma(0.375, e, 0.5), y);
}
static __device__ __noinline__ double pow_fp64(double x, double a) { return pow(x, a); }
static __device__ __noinline__ double mul_fp64(double a, double b) { return __dmul_rn(a, b); }
static __device__ __noinline__ double sqrt_fp64(double x) { return __dsqrt_rn(x); }

// the mantissa of (hi, lo) as a float in [1, 2), truncated to 23 bits
__device__ __forceinline__ float mant_f32(uint32_t lo, uint32_t hi) {
    return __uint_as_float((__funnelshift_l(lo, hi, 3) & 0x7fffffu) | 0x3f800000u);
}
// an estimate of a value in [0.5, 1] as a 24-bit fraction Y / 2^24 in [0.5, 1):
// an estimate that its error took past either end is set to the end
__device__ __forceinline__ uint32_t frac24(float y) {
    return (__float_as_uint(fmaxf(fminf(y, 0.99999994f), 0.5f)) & 0x7fffffu) | 0x800000u;
}

// 1/x as a fixed-point number, R / 2^63 in [2^62, 2^63] up to its own error (below
// 2^-9 of the result's last place).  Units: e in 2^-76, y e and y e^2 in 2^-76.
__device__ __forceinline__ uint64_t rcp_fixed(uint32_t xl, uint32_t xh) {
    float yf;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(yf) : "f"(mant_f32(xl, xh)));
    const uint32_t Y = frac24(yf), Mh = (xh & 0xfffffu) | 0x100000u;
    const int64_t E = -(int64_t)(mul_wide(xl, Y) + ((uint64_t)(Mh * Y) << 32));   // 2^76 - M Y, mod 2^64
    int64_t T = mul_hi32(E << 8, Y);
    T += ((int64_t)(int32_t)(E >> 23) * (int32_t)(T >> 23)) >> 30;
    return (uint64_t)(((int64_t)Y << 39) + (T >> 13));
}
// r / 2^53 with the sign and the exponent of 1/x
__device__ __forceinline__ double rcp_pack(uint64_t r, uint32_t xh) {
    const uint32_t rh = hi_word(r) + (0x7fc00000u - (xh & 0x7ff00000u));
    return __hiloint2double(rh | (xh & 0x80000000u), (uint32_t)r);
}

// 1/x, within 0.52 ulp
__device__ __forceinline__ double frcp(double x) {
    const uint32_t xh = __double2hiint(x), xl = __double2loint(x);
    // exponent field in [2, 2044]: 1/x normal
    if ((xh & 0x7fffffffu) - 0x00200000u >= 0x7fb00000u) return rcp_fp64(x);
    return rcp_pack((rcp_fixed(xl, xh) + 512) >> 10, xh);
}
__device__ __forceinline__ double fdiv(double a, double b) { return a * frcp(b); }

// 1/x correctly rounded, for exponent fields in [2, 2044]: s the truncated
// reciprocal, raised by one when M (2 s + 1), M the mantissa, is below 2^106, that
// is when 1/x lies above the midpoint s + 1/2 (never on it: 2 s + 1 is odd).  The
// comparison mod 2^64: the two differ by less than 2^55.  The fixed point's error may
// put s one place above the floor (1/x is then next to s, and stays) or, next to
// s + 1, one below (and is raised).
__device__ __forceinline__ double frcp_rn(double x) {
    const uint32_t xh = __double2hiint(x), xl = __double2loint(x), Mh = (xh & 0xfffffu) | 0x100000u;
    const uint64_t s = rcp_fixed(xl, xh) >> 10, m = 2 * s + 1;
    const uint64_t t = mul_wide((uint32_t)m, xl) + ((uint64_t)((uint32_t)m * Mh + hi_word(m) * xl) << 32);
    return rcp_pack(s + ((int64_t)t < 0), xh);
}

// 1/sqrt(x): z = x 4^-q in [1, 4).  Units: e in 2^-68, y e in 2^-75.
__device__ __forceinline__ double frsqrt(double x) {
    const uint32_t xh = __double2hiint(x), xl = __double2loint(x);
    if (xh - 0x00100000u >= 0x7fe00000u) return rsqrt_fp64(x);   // positive, normal
    const uint32_t odd = ~(xh >> 20) & 1u;                       // exponent - 1023 odd
    const uint64_t M = words(xl, (xh & 0xfffffu) | 0x100000u) << odd;
    const uint32_t Mh = hi_word(M), Ml = (uint32_t)M;
    float yf;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(yf) : "f"(__uint_as_float(__float_as_uint(mant_f32(xl, xh)) + (odd << 23))));
    const uint32_t Y = frac24(yf);
    const uint64_t S = mul_wide(Y, Y);
    const uint32_t Sh = hi_word(S), Sl = (uint32_t)S;
    const int64_t E = -(int64_t)((uint64_t)__umulhi(Ml, Sl) + mul_wide(Mh, Sl) + mul_wide(Ml, Sh) +
                                 ((uint64_t)(Mh * Sh) << 32));   // 2^68 - z y^2 2^68, mod 2^64
    int64_t T = mul_hi32(E << 15, Y);
    const int64_t Q = ((int64_t)(int32_t)(E >> 16) * (int32_t)(T >> 23)) >> 30;   // y e^2 in 2^-74
    T += Q + (Q >> 1);                                           // y e / 2 + 3 y e^2 / 8 in 2^-76
    const uint64_t r = (uint64_t)(((int64_t)Y << 39) + (T >> 13) + 512) >> 10;
    const int q = ((int)(xh >> 20) - 1023 - (int)odd) >> 1;
    return __hiloint2double(hi_word(r) + (uint32_t)((1021 - q) << 20), (uint32_t)r);
}

// x = z 2^(N q), z = m 2^s in [1, 2^N); Y / 2^24 the estimate of z^(-1/N)
template <int N>
struct RootSplit {
    uint32_t s, Y;
    int q;
};
template <int N>
__device__ __forceinline__ RootSplit<N> root_split(uint32_t xl, uint32_t xh) {
    static_assert(N == 2 || N == 5 || N == 7, "roots of the ideal-gas exponents");
    RootSplit<N> o;
    if (N == 2) {
        o.s = ~(xh >> 20) & 1u;
        o.q = ((int)(xh >> 20) - 1023 - (int)o.s) >> 1;
        float yf;
        asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(yf) : "f"(__uint_as_float(__float_as_uint(mant_f32(xl, xh)) + (o.s << 23))));
        o.Y = frac24(yf);
        return o;
    }
    // the exponent, offset to a non-negative number with 1023 -> N * C, by N
    // (the products are exact quotients over the 11-bit range)
    constexpr uint32_t C = N == 5 ? 205u : 147u, RCPN = N == 5 ? 52429u : 37450u;
    const uint32_t t = (xh >> 20) + (C * N - 1023u);
    const uint32_t d = (t * RCPN) >> 18;
    o.s = t - d * N;
    o.q = (int)d - (int)C;
    float lg, yf;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(lg) : "f"(mant_f32(xl, xh)));
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(yf) : "f"((lg + (float)(int)o.s) * (float)(-1. / N)));
    o.Y = frac24(yf);
    return o;
}
// y^(N-1) in 2^-64 (N = 5, 7)
template <int N>
__device__ __forceinline__ uint64_t root_pow(uint32_t Y) {
    const uint64_t A = mul_wide(Y, Y) << 16;                                       // y^2
    const uint64_t A2 = mul_wide(hi_word(A), hi_word(A)) + 2ull * hi_word(mul_wide(hi_word(A), (uint32_t)A));   // y^4
    if (N == 5) return A2;
    return mul_wide(hi_word(A2), hi_word(A)) + hi_word(mul_wide(hi_word(A2), (uint32_t)A)) +
           hi_word(mul_wide((uint32_t)A2, hi_word(A)));                            // y^6
}
// floor(a b / 2^64) up to one unit in the last place, and the next 32 bits
__device__ __forceinline__ void mul_top(uint64_t a, uint64_t b, uint32_t &w1, uint32_t &w2, uint32_t &w3) {
    const uint64_t t = mul_wide((uint32_t)a, (uint32_t)b);
    const uint64_t u = mul_wide(hi_word(a), (uint32_t)b) + hi_word(t);
    const uint64_t v = mul_wide((uint32_t)a, hi_word(b)) + (uint32_t)u;
    const uint64_t w = mul_wide(hi_word(a), hi_word(b)) + hi_word(u) + hi_word(v);
    w1 = (uint32_t)v; w2 = (uint32_t)w; w3 = hi_word(w);
}

// x^(-1/N) for N = 5, 7
template <int N>
__device__ __forceinline__ double rroot(double x) {
    const uint32_t xh = __double2hiint(x), xl = __double2loint(x);
    if (xh - 0x00100000u >= 0x7fe00000u) return pow_fp64(x, -1. / N);
    const RootSplit<N> o = root_split<N>(xl, xh);
    const uint64_t p = root_pow<N>(o.Y);
    const uint64_t yn = mul_wide(hi_word(p), o.Y << 8) + hi_word(mul_wide((uint32_t)p, o.Y << 8));   // y^N in 2^-64
    const uint64_t Z = words(xl, (xh & 0xfffffu) | 0x100000u) << (o.s + 4u);       // z in 2^-56
    uint32_t w1, w2, w3;
    mul_top(Z, yn, w1, w2, w3);                                                    // z y^N in 2^-88
    const int64_t E = -(int64_t)words(__funnelshift_l(w1, w2, 24), __funnelshift_l(w2, w3, 24));   // r in 2^-80
    const int64_t T = mul_hi32(E, o.Y);                                            // y r in 2^-72
    // y r / N: the reciprocal's 32 bits, C N = 2^32 + K, and its remainder
    constexpr uint32_t CN = N == 5 ? 0x33333334u : 0x24924925u;
    constexpr int K = N == 5 ? 4 : 3;
    int64_t D = mul_hi32(T, CN);
    D -= (int64_t)((int32_t)(D >> 32) * K);
    // (1 + N) / (2 N^2) y r^2
    constexpr int32_t C2 = N == 5 ? 0x1eb851ec : 0x14e5e0a7;                       // 0.12, 4/49 in 2^-32
    const int32_t q2 = hi_word((uint64_t)((int64_t)(int32_t)(E >> 32) * (int32_t)(T >> 24)));   // y r^2 in 2^-64
    D += (int64_t)__mulhi(q2, C2) << 8;
    const uint64_t r = (uint64_t)(((int64_t)o.Y << 39) + (D >> 9) + 512) >> 10;
    return __hiloint2double(hi_word(r) + (uint32_t)((1021 - o.q) << 20), (uint32_t)r);
}

// z^(1/N) = W (1 + a r + a (a + 1) / 2 r^2), W = z y^(N-1), a = (N-1)/N, as
// R / 2^62, R in [2^62, 2^63] up to the rounding of the caller
template <int N>
__device__ __forceinline__ uint64_t root_fixed(uint32_t xl, uint32_t xh, const RootSplit<N> &o) {
    // W in 2^-62: it may pass 2 when the estimate is high
    uint64_t W;
    const uint64_t M = words(xl, (xh & 0xfffffu) | 0x100000u);
    if (N == 2) {
        const uint64_t Z = M << (o.s + 10u);                                       // z in 2^-62
        W = mul_wide(hi_word(Z), o.Y << 8) + hi_word(mul_wide((uint32_t)Z, o.Y << 8));
    } else {
        uint32_t w1, w2, w3;
        mul_top(M << (o.s + 3u), root_pow<N>(o.Y), w1, w2, w3);                    // W in 2^-87
        W = words(__funnelshift_l(w1, w2, 7), __funnelshift_l(w2, w3, 7));
    }
    // r = 1 - W y in 2^-62
    const uint64_t t = mul_wide((uint32_t)W, o.Y), u = mul_wide(hi_word(W), o.Y) + hi_word(t);
    const int64_t E = (int64_t)(0x4000000000000000ull - ((u << 8) | ((uint32_t)t >> 24)));
    const int64_t Es = E << 17;                                                    // r in 2^-79
    int64_t g;                                                                     // a r in 2^-79
    if (N == 2) {
        g = Es >> 1;
    } else {
        constexpr uint32_t CA = N == 5 ? 0xcccccccdu : 0xdb6db6dbu;                // 4/5 + 1/(5 2^32), 6/7 - 3/(7 2^32)
        g = (int64_t)hi_word(mul_wide((uint32_t)Es, CA)) + (int64_t)(int32_t)(Es >> 32) * (int64_t)CA;
        g += N == 5 ? -(g >> 34) : (g >> 33);
    }
    // a (a + 1) / 2: 3/8 in 2^-32, 18/25 and 39/49 in 2^-31
    constexpr int32_t C2 = N == 2 ? 0x60000000 : N == 5 ? 0x5c28f5c3 : 0x65e0a72f;
    const int32_t rs = (int32_t)(E >> 15);
    const int32_t r2 = hi_word((uint64_t)((int64_t)rs * rs));                      // r^2 in 2^-62
    g += (int64_t)__mulhi(r2, C2) << (N == 2 ? 17 : 18);
    // W g in 2^-77
    const int32_t gh = (int32_t)(g >> 32);
    const int64_t Wg = (int64_t)hi_word(mul_wide(hi_word(W), (uint32_t)g)) + (int64_t)hi_word(W) * gh +
                       (((int64_t)(uint32_t)W * gh) >> 32);
    return W + (uint64_t)(Wg >> 15);
}

// x^(1/N) for N = 5, 7
template <int N>
__device__ __forceinline__ double root(double x) {
    const uint32_t xh = __double2hiint(x), xl = __double2loint(x);
    if (xh - 0x00100000u >= 0x7fe00000u) return pow_fp64(x, 1. / N);
    const RootSplit<N> o = root_split<N>(xl, xh);
    const uint64_t r = (root_fixed<N>(xl, xh, o) + 512) >> 10;
    return __hiloint2double(hi_word(r) + (uint32_t)((1022 + o.q) << 20), (uint32_t)r);
}

// sqrt(x), correctly rounded (the bits of __dsqrt_rn): s the truncated root,
// raised by one when its upper midpoint's square does not exceed the operand
// (the comparison mod 2^64: the two differ by less than 2^57)
__device__ __forceinline__ double fsqrt_rn(double x) {
    const uint32_t xh = __double2hiint(x), xl = __double2loint(x);
    if (xh - 0x00100000u >= 0x7fe00000u) return sqrt_fp64(x);
    const RootSplit<2> o = root_split<2>(xl, xh);
    const uint64_t s = root_fixed<2>(xl, xh, o) >> 10;                             // in 2^-52
    const uint64_t m = 2 * s + 1;                                                  // in 2^-53
    const uint64_t m2 = mul_wide((uint32_t)m, (uint32_t)m) + ((uint64_t)(2u * (uint32_t)m * hi_word(m)) << 32);
    const uint64_t z = (uint64_t)xl << (54u + o.s);                                // operand in 2^-106, mod 2^64
    const uint64_t r = s + ((int64_t)(z - m2) >= 0);
    return __hiloint2double(hi_word(r) + (uint32_t)((1022 + o.q) << 20), (uint32_t)r);
}

// the 106-bit product of two normal doubles, one place to the left where its
// top bit is clear, and rounded to nearest even with the carry running into
// the exponent field
__device__ __forceinline__ double mul_mantissas(uint32_t ah, uint32_t al, uint32_t bh, uint32_t bl) {
    const uint32_t mah = __funnelshift_l(al, ah, 11) | 0x80000000u, mal = al << 11, mbh = (bh & 0xfffffu) | 0x100000u;
    const uint64_t t = mul_wide(mal, bl), u = mul_wide(mah, bl) + hi_word(t);
    const uint64_t v = mul_wide(mal, mbh) + (uint32_t)u, w = mul_wide(mah, mbh) + hi_word(u) + hi_word(v);
    uint32_t wh = hi_word(w), wl = (uint32_t)w, vl = (uint32_t)v;
    uint32_t ex = (ah & 0x7ff00000u) + (bh & 0x7ff00000u) - (1023u << 20) + ((ah ^ bh) & 0x80000000u);
    if (wh < 0x100000u) {
        wh = __funnelshift_l(wl, wh, 1);
        wl = __funnelshift_l(vl, wl, 1);
        vl <<= 1;
        ex -= 0x100000u;
    }
    // remainder below the last bit (sticky in bit 0); it rounds up when
    // remainder + 2^31 - 1 + (last bit) carries
    const uint32_t rem = vl | ((uint32_t)t != 0u), half = (wl & 1u) + 0x7fffffffu;
    uint32_t rl, rh;
    asm("{\n\t.reg .u32 drop;\n\tadd.cc.u32 drop, %2, %3;\n\taddc.cc.u32 %0, %4, 0;\n\taddc.u32 %1, %5, %6;\n\t}"
        : "=r"(rl), "=r"(rh) : "r"(rem), "r"(half), "r"(wl), "r"(wh), "r"(ex));
    return __hiloint2double(rh, rl);
}
// not 0 in the top bits unless the exponent field is in [767, 1278] (2^-256 to
// 2^256): products and quotients of two such numbers are normal
__device__ __forceinline__ uint32_t out_of_window(uint32_t h) { return (h & 0x7fffffffu) - 0x2ff00000u; }

// a b, the IEEE product bit for bit; outside the window the FP64 product
__device__ __forceinline__ double xmul(double a, double b) {
    const uint32_t ah = __double2hiint(a), al = __double2loint(a), bh = __double2hiint(b), bl = __double2loint(b);
    if ((out_of_window(ah) | out_of_window(bh)) & 0xe0000000u) return mul_fp64(a, b);
    return mul_mantissas(ah, al, bh, bl);
}

static __device__ __noinline__ double div_fp64(double a, double b) { return a / b; }
// a / b correctly rounded: the quotient by the reciprocal r and its remainder's
// correction, three FP64 instructions (90 SM cycles per warp for a / b).  With r
// correctly rounded this is the IEEE quotient (P. Markstein, "Computation of
// elementary functions on the IBM RISC System/6000 processor", 1990): beside a
// midpoint of two doubles the estimate q is one of the two, half an ulp off, so the
// corrected value is off by half an ulp times |b r - 1| <= 2^-54 b (b in [1, 2)), less
// than the distance of any quotient from a midpoint, half an ulp times 2^-52 / b.
// Zero, subnormal, infinite and NaN operands and
// those outside the window, by a / b.
__device__ __forceinline__ double fdiv_rn(double a, double b) {
    const uint32_t ah = __double2hiint(a), bh = __double2hiint(b);
    if ((out_of_window(ah) | out_of_window(bh)) & 0xe0000000u) return div_fp64(a, b);
    const double r = frcp_rn(b), q = mulr(a, r);
    return fma(fma(-q, b, a), r, q);
}

}  // namespace mlh
