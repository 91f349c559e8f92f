// Pair terms of the FP64 path in 64-bit integer arithmetic: the constants a box needs, and the host
// code that forms them.  The device side is fixed64.cuh.
#pragma once
#include <cstdint>

#include "dev_types.hpp"

namespace mcg {

// Constants of one box.  Lengths are in units of the effective box Leff: max(L) / 2^sh, where the
// wrapped 64-bit displacement of a pair within reach, shifted left by sh, still fits 63 bits; or
// 2 max(L) with displacements halved, for pairs at any distance.
struct Fix64Geom {
    int sh;                  // left shift of the stored positions, hence of every displacement
    int iso;                 // equal box lengths and displacements not halved
    int up;                  // displacement = high half of (difference x ratio) << up: 2, or 1 when halved
    int64_t ratio[3];        // L[k] / max(L) in units of 2^-62
    uint64_t c2;             // (rc / Leff)^2 in units of 2^-64
    int sD;                  // rc^2 - ron^2, in units of 2^-64 Leff^2, shifted left by sD has bit 63 for its leading bit
    uint64_t rD;             // 2^126 / ((rc^2 - ron^2) / Leff^2 << sD), at most 2^63, so that a normalised
                             // rc^2 - u times it stays below 2^63: v = (rc^2 - u) / (rc^2 - ron^2)
    float Ls[3], Ll[3];      // L / 2^32 as float-float: FP32 displacement from the high words
    float in2, out2;         // FP32 r^2 below in2 lies inside ron, above out2 beyond rc (A^2)
    int emax;                // pairs whose squared distance has more leading zero bits are left to FP64
    double rc2, id2;         // rc^2 and 1 / (rc^2 - ron^2), for the pairs left to FP64
    double leff;
};

// Geometry of the pairs within rc (1 + 1e-4), switched from ron (may be 0), in a box at least 2 rc wide:
// shifted when it is at least twice the reach wide, halved otherwise.
Fix64Geom fix64_geom(const double L[3], double rc, double ron);
// Geometry of any pair of a box, without a cutoff: halved (iso: equal box lengths).
Fix64Geom fix64_geom_full(const double L[3]);

// One pair of parameter classes: el += qq Leff / r, vd += ee (w^2 - w) with w = (s / r)^6, s = si + sj.
// el comes out times Leff: a total's Coulomb sums over class pairs cancel a hundredfold, so the products
// are rounded as the reference rounds them, and the length's unit is taken out of the sum.
struct alignas(32) Fix64Pair {
    double qq, ee;       // qi qj, ei ej
    uint64_t ms;         // s^2 = ms 2^(es - 64) Leff^2, ms of at least 2^63 (0 for s = 0)
    int64_t es;
};
// Exponents of s^2 for which w is a normal double at every distance: a smaller s has no w (FP64's is below
// 2^-900), a larger one's square is infinite (FP64's from an exponent of 172 on).  A sum of sigmas that is not
// finite makes the pair's energy NaN, as FP64 does.
constexpr int FIX64_ES_MIN = -320, FIX64_ES_MAX = 300;
Fix64Pair fix64_pair(double qi, double ei, double si, double qj, double ej, double sj, double leff);

}  // namespace mcg
