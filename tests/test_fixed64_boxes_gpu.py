"""FP64 switched totals over the normalisation of the switch's constants, against the FP64 oracle.

(rc^2 - ron^2) in units of the box's squared length is held as a normalised 64-bit mantissa, so box lengths
that put it just below a power of two are where the integer switch is tightest: 26.54, 37.58, 53.0976 (the
5,000-molecule water box), 75.15 and 106.25 A at 12 and 10 A.  Tolerance as in test_fp64_pairs_gpu: a term
carries at most about 40 roundings on either side, a sum as many as its longest chain of additions.
"""
from decimal import Decimal, localcontext
from fractions import Fraction

import numpy as np
import pytest

import oracle as orc
from mc_cpp_gb300 import build, native, systems
from mc_cpp_gb300.engine import BatchChains, FFieldCUDA

pytestmark = pytest.mark.gpu
REL = 1e-13


@pytest.fixture(scope="module", autouse=True)
def _built():
    build.build()
    orc.build()
    if native.lib().mcg_device_count() < 1:
        pytest.fail("no CUDA device visible to libmcgpu.so")


def _atoms(L, box, n=3000, charges=None):
    """n charged atoms shaken off a lattice in a box of length L (times 1.25 along y for "orbic")."""
    s = systems.argon_random(n, n / L ** 3, 7)
    rng = np.random.default_rng(8)
    s.q = rng.normal(0.0, 0.3, n) if charges is None else np.full(n, charges)
    s.box = (L, L, L)
    s.set_coords(s.coords() + rng.uniform(-0.3, 0.3, (n, 3)))
    if box == "orbic":
        s.pbc_type = "orbic"
        s.box = (L, L * 1.25, L)
    return s


def _oracle(s):
    """The oracle's components, and the scale of its sums: the same system with all charges positive."""
    t = s.copy()
    t.q = np.abs(t.q)
    e, a = np.array(orc.Oracle(s, moves=False).energy()), orc.Oracle(t, moves=False).energy()
    return e, abs(a[3]) + 4 * abs(a[4])


LENGTHS = [26.54, 37.58, 53.0976, 75.15, 106.25]


@pytest.mark.parametrize("L", LENGTHS)
@pytest.mark.parametrize("box", ["cubic", "orbic"])
def test_switched_energy(L, box):
    s = _atoms(L, box, 900 if L < 30 else 3000)
    got = FFieldCUDA(s, "fp64", moves=False).getE10()
    want, scale = _oracle(s)
    assert abs(got[3] - want[3]) <= REL * scale and abs(got[4] - want[4]) <= REL * scale, (got, want, scale)


@pytest.mark.parametrize("box", ["cubic", "orbic"])
def test_batch_total(box):
    chains = [_atoms(L, box, 900 if L < 30 else 1500, charges=0.2) for L in LENGTHS]
    got = BatchChains(chains, dmax_trn=0.05, dmax_rot=1.0, seed=1).energy_fp64()
    for e, s in zip(got, chains):
        want, scale = _oracle(s)
        # a batch holds box fractions to 2^-64 and converts the coordinates once: 2^-53 L of a coordinate,
        # which moves a pair's x^12 by 12 sqrt(3) 2^-52 L / r; the closest pairs here are 1.2 A apart
        assert abs(e - want[3] - want[4]) <= (2 * REL + 21 * 2.0 ** -52 * s.box[0] / 1.2) * scale, (e, want, scale)


# Pairs closer than the 64-bit form reaches (some 2^-15 of the longest box length) in a long box, with the
# switch beginning at 0: it leaves 3 (r / rc)^4, 6e-9, of a pair's energy.  The pairs lie along x, whose
# coordinates the masters hold to 2^-53 of 30 A.
@pytest.mark.parametrize("cuton", [0.0, 10.0])
def test_batch_total_close_pairs(cuton):
    n, r, L = 40, 0.08, (30.0, 30.0, 3000.0)
    s = systems.argon_random(n, 0.0213, 3)
    s.pbc_type, s.box, s.cuton = "orbic", L, cuton
    s.q, s.eps = np.full(n, 0.2), np.zeros(n)
    z = np.repeat(np.arange(n // 2) * 140.0 - 1400.0, 2)
    s.set_coords(np.stack([np.tile([3.0, 3.0 + r], n // 2), np.zeros(n), z], 1))
    got = BatchChains([s], dmax_trn=0.05, dmax_rot=1.0, seed=1).energy_fp64()[0]
    want, scale = _oracle(s)
    assert abs(got - want[3] - want[4]) <= (2 * REL + 2 * 2.0 ** -52 * 30.0 / r) * scale, (got, want, scale)


# One pair in boxes of up to a million A: what the box fractions' unit is worth grows with the box, so close
# pairs are left to FP64 there.  The exact value in rationals; beside it the FP64 form carries 3 roundings of r^2
# (half of each counts), 1 of 1/r, 2 of x = s / r, 12 times those, and 6 more: 60, with the switch's own
# (8 roundings, none of them cancelling at these distances) and the totals' factors 72.
@pytest.mark.parametrize("L", [30.0, 100.0, 1e3, 1e4, 1e5, 1e6])
@pytest.mark.parametrize("shape", ["cubic", "slab"])
@pytest.mark.parametrize("cut", ["full", "switch"])
def test_one_pair_in_a_large_box(L, shape, cut):
    K, rng = 332.0716 * 418.4, np.random.default_rng(11)
    for r in (1.1, 1.7, 2.5, 3.3, 4.1, 10.7):
        s = systems.argon_random(2, 0.0213, 3)
        v = rng.normal(size=3)
        a = rng.uniform(-3.0, 3.0, 3)
        s.set_coords(np.stack([a, a + r * v / np.linalg.norm(v)]))
        s.pbc_type, s.box = ("cubic", (L, L, L)) if shape == "cubic" else ("orbic", (30.0, L, 31.0))
        s.cut_mode, s.q = cut, np.array([0.4, -0.3])
        got = FFieldCUDA(s, "fp64", moves=False).getE10()
        d2 = sum((Fraction(p) - Fraction(q)) ** 2 for p, q in zip(*s.coords()))
        S = Fraction(1)
        if cut == "switch" and d2 > 100:
            S = (144 - d2) ** 2 * (144 + 2 * d2 - 300) / Fraction(44) ** 3
        with localcontext() as c:
            c.prec = 50
            root = (Decimal(d2.numerator) / Decimal(d2.denominator)).sqrt()
        e = np.sqrt(s.eps * 418.4)
        x6 = (Fraction(s.sig[0]) + Fraction(s.sig[1])) ** 6 / d2 ** 3
        elec = Fraction(s.q[0]) * Fraction(s.q[1]) * Fraction(K) * S / Fraction(root)
        vdw = 4 * Fraction(e[0]) * Fraction(e[1]) * (x6 * x6 - x6) * S
        # (x6 - 1) can cancel: its scale is that of x^12 + x^6
        scale = float(4 * Fraction(e[0]) * Fraction(e[1]) * (x6 * x6 + x6) * S)
        assert abs(got[3] - float(elec)) <= 72 * 2.0 ** -53 * abs(float(elec)), (r, got[3], float(elec))
        assert abs(got[4] - float(vdw)) <= 72 * 2.0 ** -53 * scale, (r, got[4], float(vdw), scale)


# sigmas whose powers leave the range of a double: a tiny one's x^6 is 0, a huge one's energy is not finite, nor is
# that of one that is not finite itself; 200 charges leave the class table
@pytest.mark.parametrize("sig", [1e-30, 1e-47, 1e-60, 1e-155, 1e-300, 1e60, 1e200, float("inf"), float("nan")])
@pytest.mark.parametrize("cut", ["full", "switch"])
@pytest.mark.parametrize("classes", [1, 200])
def test_extreme_sigma(sig, cut, classes):
    n = 300
    s = _atoms(30.0, "cubic", n)
    s.q = np.resize(np.linspace(-0.4, 0.4, classes) if classes > 1 else [0.3], n)
    s.cut_mode, s.sig = cut, s.sig.copy()
    s.sig[:] = sig
    got = FFieldCUDA(s, "fp64", moves=False).getE10()
    want, scale = _oracle(s)
    assert abs(got[3] - want[3]) <= REL * abs(_oracle_elec(s)), (got, want)
    assert np.isfinite(got[4]) == np.isfinite(want[4]), (got, want)
    if np.isfinite(want[4]):
        assert abs(got[4] - want[4]) <= REL * abs(want[4]) + 1e-250, (got, want)


def _oracle_elec(s):
    t = s.copy()
    t.q = np.abs(t.q)
    return orc.Oracle(t, moves=False).energy()[3]


@pytest.mark.parametrize("sig", [1e-60, 1e-300])
def test_extreme_sigma_batch(sig):
    s = _atoms(30.0, "cubic", 300, charges=0.2)
    s.sig = np.full(300, sig)
    got = BatchChains([s], dmax_trn=0.05, dmax_rot=1.0, seed=1).energy_fp64()[0]
    want, _ = _oracle(s)
    assert abs(got - want[3] - want[4]) <= (2 * REL + 2 * 2.0 ** -52 * 30.0 / 1.2) * abs(want[3]), (got, want)
