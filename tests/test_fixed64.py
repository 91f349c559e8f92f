"""The 64-bit integer pair terms (csrc/fixed64.cuh) restated in Python integers, against exact rationals.

The bounds are the roundings of each form: Y keeps units of 2^-59 of 1 and the iteration's remainder
(5/2 d^3 for a seed within d = 2^-22), w = (s Y)^6 truncates one unit of 2^-60 twice before it is cubed
and up to 3 units of it twice after, and the switch keeps 2^-57 of itself beside what two units of the squared distance do to it.
"""
import math
import random
from fractions import Fraction as Fr

import numpy as np
import pytest

M64 = (1 << 64) - 1


def hi(a, b):
    assert 0 <= a <= M64 and 0 <= b <= M64
    ah, al, bh, bl = a >> 32, a & 0xFFFFFFFF, b >> 32, b & 0xFFFFFFFF
    r = ah * bh + ((ah * bl) >> 32) + ((al * bh) >> 32)
    assert 0 <= ((a * b) >> 64) - r <= 3
    return r


def s32(v):
    v &= 0xFFFFFFFF
    return v - (1 << 32) if v >> 31 else v


def dist2(d):
    s2 = s1 = t = 0
    for v in d:
        l = s32(v)
        h = (v >> 32) + (l < 0)
        assert -(1 << 31) <= h < 1 << 31 and h * (1 << 32) + l == v
        s2, s1, t = s2 + h * h, s1 + h * l, t + ((l * l) >> 32)
        assert abs(s1) < 1 << 63 and t < 1 << 32
    s1 += t >> 1
    H = s2 + (s1 >> 31)
    assert 0 <= H <= M64
    return H >> 32, H & 0xFFFFFFFF, (s1 << 1) & 0xFFFFFFFF


def terms(uh, um, ul, seed_error, ms):
    e2 = (32 - uh.bit_length()) & ~1
    m = ((uh << 64 | um << 32 | ul) >> (32 - e2)) & M64
    f = np.float32(np.float32(1) / np.sqrt(np.float32(m >> 32)) * np.float32(1 + seed_error))
    y0 = min(int(np.float32(f * np.float32(2.0 ** 46))), 1 << 31)
    e = (1 << 60) - hi(m, y0 * y0)
    es = e >> 9
    assert -(1 << 31) <= es < (1 << 31)
    c = e + ((3 * ((es * es) >> 42)) >> 2)
    Y = (y0 << 32) + ((y0 * (c >> 32) + ((y0 * (c & 0xFFFFFFFF)) >> 32)) << 3)
    w1 = (Y * Y) >> 64 << 1
    x = (w1 * ms) >> 64
    assert 1 << 59 <= x < 1 << 63 and (1 << 62) - (1 << 8) <= Y <= (1 << 63) + (1 << 8)
    lx = 63 - x.bit_length()
    x <<= lx
    x6 = hi(x, hi(x, x) << 2)
    assert 1 << 59 <= x6 < 1 << 63
    return Y, x6, e2, lx


def test_inverse_powers():
    rng = random.Random(1)
    worst_y = worst_w = 0.0
    for _ in range(4000):
        r = 0.49998 * 10 ** rng.uniform(-3.3, 0)    # fractions of Leff up to the reach
        v = [rng.gauss(0, 1) for _ in range(3)]
        n = math.sqrt(sum(x * x for x in v))
        d = [int(x / n * r * 2 ** 64) for x in v]
        u = Fr(sum(x * x for x in d), 1 << 128)
        uu = dist2(d)
        if 32 - uu[0].bit_length() > 29:
            continue
        ms = rng.choice([1 << 63, M64, rng.randrange(1 << 63, 1 << 64)])      # s^2 = ms 2^-64
        Y, x6, e2, lx = terms(*uu, rng.choice([-1, 1]) * 2.0 ** -22, ms)
        y = Fr(Y, 1 << 62) * (1 << (e2 // 2))
        worst_y = max(worst_y, abs(float(y * y * u - 1)) / 2)
        worst_w = max(worst_w, abs(float(Fr(x6, 1 << 57) * Fr(1 << (3 * e2), 1 << (3 * lx)) * u ** 3 / Fr(ms, 1 << 64) ** 3 - 1)))
    assert worst_y < 2.0 ** -57 and worst_w < 2.0 ** -55.5, (math.log2(worst_y), math.log2(worst_w))


@pytest.mark.parametrize("m", [1 << 62, (1 << 62) + 1, (1 << 63) - 1, 1 << 63, M64])
def test_mantissa_ends(m):
    for s in (-1, 0, 1):
        Y, _, e2, _ = terms(m >> 32, m & 0xFFFFFFFF, 0, s * 2.0 ** -22, 1 << 63)
        assert e2 == 0 and abs(float(Fr(Y, 1 << 62) ** 2 * Fr(m, 1 << 64) - 1)) < 2.0 ** -56.5


@pytest.mark.parametrize("L", [24.0, 26.0, 34.4, 49.69, 100.0, 143.3])
@pytest.mark.parametrize("ron", [0.0, 5.0, 10.0, 11.9])
def test_switch(L, ron):
    rc, rng, sh, sD = 12.0, random.Random(2), 0, 0
    while sh < 20 and rc * 1.0001 * 2 ** (sh + 1) <= 0.5 * L:
        sh += 1
    l2 = (Fr(L) / 2 ** sh) ** 2
    D = Fr(rc) ** 2 - Fr(ron) ** 2
    c2, dq = int(Fr(144) / l2 * 2 ** 64), D / l2 * 2 ** 64
    span = min(Fr(144) / l2 * 2 ** 64, dq * (1 + Fr(1, 256)))
    while sD < 63 and span * 2 ** (sD + 1) < 2 ** 64:
        sD += 1
    rD = min(M64, int(Fr(2 ** 126) / (dq * 2 ** sD)))
    unit = float(l2 / D) * 2.0 ** -64
    for _ in range(500):
        uh = int(Fr(rng.uniform(ron, 12.001)) ** 2 / l2 * 2 ** 64)
        dl = c2 - uh if uh < c2 else 0
        ld = 64 - dl.bit_length()
        v = hi((dl << (ld & 63)) & M64, rD)
        if ld < sD or (ld == sD and v > 1 << 62):
            ld, v = sD, 1 << 62
        back = ld - sD
        assert v << 1 <= M64
        v2 = hi(v << 1, v << 1)
        S = hi(v2, 3 * (1 << 62) - ((v << 1) >> (back & 63)))
        V = min(max((Fr(144) - Fr(uh, 2 ** 64) * l2) / D, 0), 1)
        want = V * V * (3 - 2 * V)
        assert abs(float(Fr(S, 2 ** 60) / 4 ** back - want)) <= float(want) * 2.0 ** -57 + 12 * float(V) * unit + 12 * unit * unit
