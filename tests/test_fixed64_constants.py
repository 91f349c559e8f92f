"""The constants of the 64-bit integer pair terms as the library forms them (csrc/fixed64.cpp, compiled here),
with the switch of csrc/fixed64.cuh restated in Python integers over the whole range of their normalisation.

rc^2 - ron^2 in units of Leff^2 is normalised to a 64-bit mantissa, so its place between two powers of two
depends on the box length; the lengths here put it at and near both ends, for shifted and halved geometries.
Bound of the switch S = v^2 (3 - 2 v): a product of high halves is at most 3 units low, v is at least 2^61 units,
v^2 2^60 and S 2^59, so 2 (3 2^-61) + 3 2^-60 for v^2, as much again at most for 3 - 2 v and 3 2^-59 for S: 2^-56
together; beside it what one unit of u and one of rc^2 do to v.
"""
import math
import os
import random
import shutil
import subprocess
from fractions import Fraction as Fr

import pytest

from test_fixed64 import M64, dist2, hi

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "mc_cpp_gb300", "csrc")
MAIN = r"""
#include <cstdio>
#include "fixed64.hpp"
int main() {
    double L[3], rc, ron;
    while (std::scanf("%la %la %la %la %la", &L[0], &L[1], &L[2], &rc, &ron) == 5) {
        const mcg::Fix64Geom G = mcg::fix64_geom(L, rc, ron);
        std::printf("%d %d %d %llu %d %llu %a %d\n", G.sh, G.iso, G.up, (unsigned long long)G.c2, G.sD, (unsigned long long)G.rD, G.leff, G.emax);
    }
}
"""


@pytest.fixture(scope="module")
def geoms(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("g++ not found")
    tmp = str(tmp_path_factory.mktemp("fixed64"))
    src, exe = os.path.join(tmp, "main.cpp"), os.path.join(tmp, "geoms")
    with open(src, "w") as f:
        f.write(MAIN)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-I" + CSRC, src, os.path.join(CSRC, "fixed64.cpp"), "-o", exe])

    def get(cases):
        text = "".join("%s\n" % " ".join(float(v).hex() for v in c) for c in cases)
        out = subprocess.run([exe], input=text, stdout=subprocess.PIPE, text=True, check=True).stdout.split("\n")
        return [(int(a), int(b), int(c), int(d), int(e), int(f), float.fromhex(g), int(h)) for a, b, c, d, e, f, g, h in
                (line.split() for line in out if line)]
    return get


MANTISSAS = [0.5 * (1 + 2.0 ** -40), 0.5001, 0.51, 0.6, 0.75, 0.9, 0.99, 0.9960, 0.9962, 0.998, 0.9999, 1 - 2.0 ** -40]


def _boxes(rc, ron):
    """Cubic box lengths that put (rc^2 - ron^2) / Leff^2 at these mantissas: every power of two and
    shift; fix64_geom takes the ones whose shift is its own."""
    out = []
    for m in MANTISSAS:
        for k in range(0, 30):
            leff = math.sqrt((rc * rc - ron * ron) / m * 2.0 ** k)
            for sh in range(0, 6):
                L = leff * 2 ** sh
                if 2 * rc <= L < 400.0:
                    out.append((L, L, L, rc, ron))
    return out


def _check_switch(case, g, rng, samples):
    sh, iso, up, c2, sD, rD, leff, _ = g
    rc, ron = Fr(case[3]), Fr(case[4])
    l2 = Fr(leff) ** 2
    D = rc * rc - ron * ron
    unit = float(l2 / D) * 2.0 ** -64
    near = [float(ron) * (1 - 4e-5), float(ron)] + [math.sqrt(max(float(rc * rc - D / 2 ** k) * (1 + s), 0.0)) for k in range(0, 5)
                                                  for s in (-1e-3, -1e-9, 1e-9, 1e-3)]
    near += [rng.uniform(float(ron) * 0.99995, float(rc) * 1.0001) for _ in range(samples)]
    for r in near:
        u = Fr(r) ** 2 / l2 * 2 ** 64
        if u >= 1 << 64:
            continue
        uh = int(u)
        dl = c2 - uh if uh < c2 else 0
        ld = 64 - dl.bit_length()
        v = hi((dl << (ld & 63)) & M64, rD)
        if ld < sD or (ld == sD and v > 1 << 62):
            ld, v = sD, 1 << 62
        back = ld - sD
        v2 = hi((v << 1) & M64, (v << 1) & M64)
        S = hi(v2, 3 * (1 << 62) - (((v << 1) & M64) >> (back & 63)))
        V = min(max((rc * rc - Fr(uh, 2 ** 64) * l2) / D, 0), 1)
        want = V * V * (3 - 2 * V)
        tol = float(want) * 2.0 ** -56 + 12 * float(V) * unit + 12 * unit * unit
        assert abs(float(Fr(S, 2 ** 60) / 4 ** back - want)) <= tol, (case, r, float(V), float(Fr(S, 2 ** 60) / 4 ** back), float(want))


@pytest.mark.parametrize("rc,ron", [(12.0, 0.0), (12.0, 5.0), (12.0, 10.0), (12.0, 11.9), (12.0, 11.999), (9.0, 8.95), (9.0, 0.5)])
def test_switch_over_the_normalisation(geoms, rc, ron):
    rng = random.Random(3)
    cases = _boxes(rc, ron) + [(L, L * 1.25, L * 2.0, rc, ron) for L, _, _, _, _ in _boxes(rc, ron)[::7]]
    seen = set()
    for case, g in zip(cases, geoms(cases)):
        seen.add((g[0], g[1]))
        _check_switch(case, g, rng, 6)
    assert len(seen) >= 4, seen     # several shifts, cubic and not


# boxes too small for the shift have their displacements halved: Leff is fixed there, and ron moves the mantissa
@pytest.mark.parametrize("L", [24.0, 24.002])
def test_switch_over_the_normalisation_halved(geoms, L):
    rng = random.Random(4)
    cases = []
    for m in MANTISSAS:
        for k in range(2, 12):
            D = m * 2.0 ** -k * 4 * L * L
            if 0 < D <= 144.0:
                cases.append((L, L, L, 12.0, math.sqrt(144.0 - D)))
    for case, g in zip(cases, geoms(cases)):
        assert g[:3] == (0, 0, 1)
        _check_switch(case, g, rng, 20)


# 64-bit geometry of the water boxes of 5000, 5010 and 14180 molecules, and lengths where the leading bits are all ones
@pytest.mark.parametrize("L", [26.54, 37.58, 53.0976, 53.133, 75.15, 106.25])
def test_switch_of_common_boxes(geoms, L):
    case = (L, L, L, 12.0, 10.0)
    _check_switch(case, geoms([case])[0], random.Random(5), 2000)


# Pairs that the 64-bit form keeps: their distance from positions rounded to 2^-64 of the box, against the exact
# one.  Each component is off by a unit of each position (and by the units its scaling drops), at most 2^-53 of r
# in each of three, so r^2 by at most 2 sqrt(3) 2^-53 3.
@pytest.mark.parametrize("L", [(30.0, 30.0, 30.0), (100.0, 100.0, 100.0), (1e3, 1e3, 1e3), (9e4, 9e4, 9e4), (40.0, 40.0, 700.0), (31.0, 5e3, 47.0)])
def test_close_limit(geoms, L):
    sh, iso, up, _, _, _, leff, emax = geoms([(*L, 12.0, 10.0)])[0]
    rng, kept = random.Random(6), 0
    for _ in range(3000):
        a = [rng.uniform(-5, 5) for _ in range(3)]
        v = [rng.gauss(0, 1) for _ in range(3)]
        r = 12.0 * 10 ** rng.uniform(-4, 0) / math.sqrt(sum(x * x for x in v))
        b = [p + x * r for p, x in zip(a, v)]
        exact = sum((Fr(q) - Fr(p)) ** 2 for p, q in zip(a, b))
        d = [round(Fr(q) / Fr(l) * 2 ** 64) - round(Fr(p) / Fr(l) * 2 ** 64) for p, q, l in zip(a, b, L)]
        d = [x << sh for x in d]
        if not iso:
            d = [((x * int(Fr(l) / Fr(max(L)) * 2 ** 62)) >> 64) << up for x, l in zip(d, L)]
        uh, um, ul = dist2(d)
        if (32 - uh.bit_length()) & ~1 > emax:
            continue
        kept += 1
        u = Fr(uh << 64 | um << 32 | ul, 1 << 96) * Fr(leff) ** 2
        assert abs(float(u / exact - 1)) <= 6 * math.sqrt(3) * 2.0 ** -53, (a, b, float(exact))
    assert (kept > 50) == (math.ldexp(leff, -emax // 2 - 1) < 11.0), kept     # some pairs are kept wherever any is in reach
