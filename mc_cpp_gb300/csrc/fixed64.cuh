// Pair terms of the FP64 path in 64-bit integer arithmetic.
//
// GB300 issues one FP64 warp instruction per scheduler every 64 cycles (76 with several warps), and
// a full 64 x 64-bit integer product about every 22.  A pair's distance, inverse square root, powers
// and switch therefore run on 64-bit integers, which carry more bits than a double's 53, and only
// the products with the pair's parameters and the sums (three FMAs) are FP64.
//
// * Positions are box fractions in units of 2^-64, so unsigned subtraction wraps to the minimum
//   image exactly; the conversion from the FP64 masters keeps the quotient's remainder, so a position
//   is off by at most one unit (5e-18 A in a 100 A box), far below the master's own spacing.  They
//   are stored shifted left by the geometry's sh: a difference of two is then the displacement shifted,
//   and right as a signed number for pairs within reach.  Without a cutoff, or in a box that does not
//   hold the cutoff sphere, displacements are halved instead.
// * u = r^2 is kept to 95 bits and normalised to a 64-bit mantissa m by an even shift e2 (u = m 2^-e2
//   in units of Leff^2 2^-64).
// * Y = 1 / sqrt(m): an FP32 estimate (relative error below 2^-22), then one step of the third-order
//   Householder iteration for y^-2 - m; the error is below 2^-58.
// * w = (s / r)^6 = (s^2 Y^2)^3 by four products, with s^2 = (sig_i + sig_j)^2 given to 64 bits: off by
//   at most 2^-55 and 2^-54 in its rounding to a double (12 multiplications of a rounded quotient reach
//   2^-49).  Rounding s^6 and s^12 to doubles instead would be an error common to all pairs of two classes.
// * The switch is v^2 (3 - 2 v) with v = (rc^2 - u) / (rc^2 - ron^2) clamped to [0, 1] (the
//   reference's polynomial in another variable), to 2^-56 of itself (beside u's own last place).
// Totals against 113-bit sums, relative (FP64 pair terms in brackets).  Switched, 12 and 10 A, over 24 boxes of 28.6 to
// 60 A on both sides of the switch's normalisation, RMS: 2,400 water atoms in cubic boxes Coulomb 4.5e-16 (3.0e-15),
// Lennard-Jones 2.2e-16 (3.8e-16), orthorhombic 1.1e-15 (3.1e-15) and 0.9e-16 (1.2e-16); 500 to 1,500 argon atoms
// 1.2e-16 (3.4e-16) and 1.1e-16 (7.4e-16).  Full mode, 60 boxes of 24 to 60 A: water Coulomb (median: some totals nearly
// cancel) 3.5e-16 (5.3e-16) and 8.3e-16 (1.6e-15), Lennard-Jones RMS 0.9e-16 (1.0e-16) and 0.9e-16 (2.8e-16); argon
// 1.0e-16 (3.0e-16) and 1.0e-16 (1.9e-16).
// A pair closer than some 2^-11 of a box length (0.05 A in a box of 100 A; the geometry's emax), where the
// positions' unit would tell, is left to the caller.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "fixed64.hpp"

namespace mcg {

// x / L modulo 1 in units of 2^-64, shifted left by sh: q = fl(x rL), its distance to the nearest
// integer is exact, and the remainder x - q L is exact before its own (relative) rounding.
__device__ __forceinline__ unsigned long long to_fixed64(double x, double L, double rL, int sh) {
    const double q = __dmul_rn(x, rL);
    const double lo = fma(-q, L, x) * rL;
    return ((unsigned long long)__double2ll_rn((q - rint(q)) * 18446744073709551616.0) +
            (unsigned long long)__double2ll_rn(lo * 18446744073709551616.0)) << sh;
}

// v 2^scale as a double, rounded to nearest (ties up), for v of at least 2^63
__device__ __forceinline__ double fix64_norm_to_double(unsigned long long v, int scale) {
    const unsigned long long r = (v >> 11) + ((v >> 10) & 1ull);
    return __longlong_as_double((long long)(((unsigned long long)(1085 + scale) << 52) + r));
}

// the same for any v (0 for v = 0)
__device__ __forceinline__ double fix64_to_double(unsigned long long v, int scale) {
    const int lz = __clzll((long long)v);
    return lz == 64 ? 0.0 : fix64_norm_to_double(v << (lz & 63), scale - lz);
}

// high half of a 64 x 64-bit product, at most 3 below it (the two cross products are truncated and the
// low one left out): five instructions
__device__ __forceinline__ unsigned long long fix64_mulhi(unsigned long long a, unsigned long long b) {
    const unsigned ah = (unsigned)(a >> 32), al = (unsigned)a, bh = (unsigned)(b >> 32), bl = (unsigned)b;
    return (unsigned long long)ah * bh + __umulhi(ah, bl) + __umulhi(al, bh);
}

// v = ms 2^(es - 64) with ms of at least 2^63 for a v that is not negative, its exponent within the limits of
// fix64_pair; false when v is not finite
__device__ __forceinline__ bool fix64_mantissa(double v, unsigned long long& ms, int& es) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    const int e = (int)(b >> 52);
    es = e - 1022;
    ms = es < FIX64_ES_MIN ? 0ull : (b << 11) | (1ull << 63);
    es = min(es, FIX64_ES_MAX);
    return e < 2047;
}

struct Fix64Dist {
    unsigned hi, mid, lo;   // u = (hi 2^64 + mid 2^32 + lo) 2^-96 Leff^2
};

// Squared distance of two positions from their difference (b - a).  A displacement is split as
// h 2^32 + l with both halves signed, so its square needs no absolute value; |h| and the sums stay
// below 2^31 and 2^63 because the displacement's length is below 2^63 (halved: its components at most
// 2^62).  ISO: equal box lengths, and the displacement as it is, or halved (HALF); else scaled by the
// box's ratios, halved or not as the geometry says.
template <bool ISO, bool HALF = false>
__device__ __forceinline__ Fix64Dist fix64_dist2(const Fix64Geom& G, unsigned long long dx, unsigned long long dy,
                                                 unsigned long long dz) {
    unsigned long long s2 = 0;
    long long s1 = 0;
    unsigned t = 0;
    const unsigned long long d3[3] = {dx, dy, dz};
#pragma unroll
    for (int k = 0; k < 3; k++) {
        long long d = (long long)d3[k];
        if (!ISO) d = __mul64hi(d, (long long)G.ratio[k]) << G.up;
        else if (HALF) d >>= 1;
        const int l = (int)d, h = (int)(d >> 32) + (int)((unsigned)l >> 31);
        s2 += (unsigned long long)((long long)h * h);
        s1 += (long long)h * l;
        t += (unsigned)__mulhi(l, l);
    }
    s1 += t >> 1;                                    // units of 2^-95
    const unsigned long long H = s2 + (unsigned long long)(s1 >> 31);
    return Fix64Dist{(unsigned)(H >> 32), (unsigned)H, (unsigned)s1 << 1};
}

template <bool ISO, bool HALF = false>
__device__ __forceinline__ Fix64Dist fix64_dist2(const Fix64Geom& G, const ulonglong4_32a& a, const ulonglong4_32a& b) {
    return fix64_dist2<ISO, HALF>(G, b.x - a.x, b.y - a.y, b.z - a.z);
}

// w = (s / r)^6 for s^2 = ms 2^(es - 64) Leff^2 (ms of at least 2^63, or 0), and ys = Leff / r and ws = w
// times the switch factor (1 unless sw, 0 beyond rc).  False when the pair is too close for the form.
__device__ __forceinline__ bool fix64_terms(const Fix64Geom& G, const Fix64Dist& u, bool sw, unsigned long long ms, int es,
                                            double& ys, double& w, double& ws) {
    const int e2 = __clz((int)u.hi) & ~1;
    const unsigned mh = __funnelshift_l(u.mid, u.hi, e2), ml = __funnelshift_l(u.lo, u.mid, e2);
    const unsigned long long m = (unsigned long long)mh << 32 | ml;
    // 1 / sqrt of the mantissa in [1/4, 1): Y in (1, 2], units of 2^-62
    const float f = rsqrtf(__uint2float_rn(mh));
    const unsigned y0 = __float2uint_rz(fminf(f * 70368744177664.0f, 2147483648.0f));   // units of 2^-30
    const unsigned long long t = (unsigned long long)y0 * y0;
    const long long e = (long long)((1ull << 60) - fix64_mulhi(m, t));                   // 1 - m y0^2, units of 2^-60
    const int e9 = (int)(e >> 9);
    const long long c = e + (3 * (((long long)e9 * e9) >> 42) >> 2);                     // e/2 + 3/8 e^2, units of 2^-61
    const long long corr = (long long)y0 * (int)(c >> 32) + (long long)__umulhi(y0, (unsigned)c);
    const unsigned long long Y = ((unsigned long long)y0 << 32) + (unsigned long long)(corr << 3);
    const int k = e2 >> 1;
    const unsigned long long W1 = __umul64hi(Y, Y) << 1;            // y^2, units of 2^-61
    unsigned long long X = __umul64hi(W1, ms);                       // (s / r)^2, units of 2^(es + 2k - 61)
    const int lx = __clz((int)(X >> 32)) - 1, ex = es + 2 * k - lx;  // leading bit from 59 .. 62 to 62
    X <<= lx & 63;
    const unsigned long long X4 = fix64_mulhi(X, X);                 // units of 2^(2 ex - 58)
    const unsigned long long X6 = fix64_mulhi(X, X4 << 2);           // units of 2^(3 ex - 57)
    const int lw = __clz((int)(X6 >> 32)) - 1;                       // leading bit from 59 .. 62 to 62
    const unsigned long long wn = X6 << (lw & 63);
    w = ms ? __longlong_as_double((long long)(((unsigned long long)(1084 - 57 + 3 * ex - lw) << 52) + ((wn + 512) >> 10))) : 0.0;
    ys = __longlong_as_double((long long)(((unsigned long long)(1022 + k) << 52) + ((Y + 512) >> 10)));
    ws = w;
    if (sw) {
        // v and v^2 with a shift of their own, so the switch keeps its relative accuracy near rc.  rD is at
        // most 2^63 (fix64_geom), so v stays below 2^63 and v << 1 within 64 bits, at every box length
        const unsigned long long uh = (unsigned long long)u.hi << 32 | u.mid;
        const unsigned long long dl = uh < G.c2 ? G.c2 - uh : 0ull;
        int ld = __clzll((long long)dl);
        unsigned long long v = fix64_mulhi(dl << (ld & 63), G.rD);   // units of 2^-62 2^(sD - ld)
        if (ld < G.sD || (ld == G.sD && v > (1ull << 62))) { ld = G.sD; v = 1ull << 62; }   // inside ron
        const int back = ld - G.sD;
        const unsigned long long v2 = fix64_mulhi(v << 1, v << 1);   // units of 2^-62 2^(-2 back)
        const unsigned long long S = fix64_mulhi(v2, 3ull * (1ull << 62) - (v << 1 >> (back & 63)));   // 2^-60 2^(-2 back)
        const double s = fix64_to_double(S, -60 - 2 * back);
        ys *= s;
        ws *= s;
    }
    return e2 <= G.emax;
}

}  // namespace mcg
