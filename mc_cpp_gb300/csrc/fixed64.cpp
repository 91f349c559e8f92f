// Host side of the 64-bit integer pair terms (fixed64.hpp): each constant rounded once from extended
// precision.
#include "fixed64.hpp"

#include <algorithm>
#include <cmath>

namespace mcg {

namespace {
constexpr long double TWO64L = 18446744073709551616.0L;

uint64_t clamp64(long double v) { return v >= TWO64L ? ~0ull : (v <= 0.0L ? 0ull : (uint64_t)v); }

// A displacement's component is off by the positions' unit, or by the units that its scaling drops.  Pairs so
// close that this passes 2^-53 of their distance are left to FP64, whose differences of nearby coordinates
// are exact: r^-12 is off by some 5 times that share (RMS), 6e-16, where the FP64 form's is off by 1.1e-15.
// A squared distance with e leading zero bits, e even, is at least 2^-(e + 2) of Leff^2.  Cubic boxes of 100 A
// switched, 60 A in full mode: 0.05 and 0.06 A; a box of 10,000 A: 4.9 A.
int close_limit(const Fix64Geom& G, double lmax) {
    const double unit = std::ldexp(std::max(lmax, G.iso ? G.leff : std::ldexp(G.leff, G.up)), -64);
    int e = 28;
    while (e >= 0 && std::ldexp(G.leff, -(e / 2 + 1)) < std::ldexp(unit, 53)) e -= 2;
    return e;
}
}  // namespace

Fix64Geom fix64_geom_full(const double L[3]) {
    Fix64Geom G{};
    const double lmax = std::max(L[0], std::max(L[1], L[2]));
    G.iso = L[0] == L[1] && L[1] == L[2];
    G.up = 1;
    G.leff = 2.0 * lmax;
    for (int k = 0; k < 3; k++) {
        G.ratio[k] = (int64_t)clamp64((long double)L[k] / (long double)lmax * (TWO64L / 4));
        const double ls = L[k] / 4294967296.0;
        G.Ls[k] = (float)ls;
        G.Ll[k] = (float)(ls - (double)G.Ls[k]);
    }
    G.emax = close_limit(G, lmax);
    return G;
}

Fix64Geom fix64_geom(const double L[3], double rc, double ron) {
    const double reach = rc * (1.0 + 1e-4);
    Fix64Geom G = fix64_geom_full(L);
    const double lmax = std::max(L[0], std::max(L[1], L[2])), lmin = std::min(L[0], std::min(L[1], L[2]));
    if (2.0 * reach <= lmin) {
        // reach / lmin 2^sh <= 1/2, so a displacement within reach stays within 63 bits after the shift
        while (G.sh < 20 && reach * std::ldexp(1.0, G.sh + 1) <= 0.5 * lmin) G.sh++;
        G.up = 2;
        G.leff = std::ldexp(lmax, -G.sh);
    } else {
        G.iso = 0;   // halved, by the general form
    }
    G.emax = close_limit(G, lmax);
    const long double l2 = (long double)G.leff * (long double)G.leff;
    const long double c2 = (long double)rc * rc, d = c2 - (long double)ron * ron;
    G.c2 = clamp64(c2 / l2 * TWO64L);
    const long double dq = d / l2 * TWO64L;            // rc^2 - ron^2 in units of 2^-64
    while (G.sD < 63 && std::ldexp(dq, G.sD + 1) < TWO64L) G.sD++;
    G.rD = clamp64(std::ldexp(1.0L, 126) / std::ldexp(dq, G.sD));
    G.rc2 = rc * rc;
    G.id2 = 1.0 / (G.rc2 - ron * ron);
    G.in2 = (float)(ron * ron * (1.0 - 1e-4));
    G.out2 = (float)(rc * rc * (1.0 + 1e-4));
    return G;
}

Fix64Pair fix64_pair(double qi, double ei, double si, double qj, double ej, double sj, double leff) {
    const long double s = ((long double)si + (long double)sj) / (long double)leff;
    if (!std::isfinite(s)) return Fix64Pair{qi * qj, std::nan(""), 0, 0};
    int es = 0;
    const long double f = std::frexp(s * s, &es);   // in [1/2, 1)
    return Fix64Pair{qi * qj, ei * ej, es < FIX64_ES_MIN ? 0 : clamp64(f * TWO64L), std::min(es, FIX64_ES_MAX)};
}

}  // namespace mcg
