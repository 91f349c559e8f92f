"""FP64 pair arithmetic and energy kernels where they can go wrong, against the FP64 oracle.

Tolerance: a pair term carries at most about 40 roundings on either side (twelve of them through
x^12), and a sum of N terms as many as its longest chain of additions, so 1e-13 of the sum of the
terms' magnitudes bounds both for the sizes here.  Only totals are visible, so the magnitude is
taken from the oracle's energies of the attractive and repulsive parts, |elec| + |vdw| of the same
system with all charges made positive.
"""
from decimal import Decimal, localcontext

import numpy as np
import pytest

import oracle as orc
from mc_cpp_gb300 import build, native, systems
from mc_cpp_gb300.engine import BatchChains, FFieldCUDA

pytestmark = pytest.mark.gpu
REL = 1e-13
KCAL = 418.4


@pytest.fixture(scope="module", autouse=True)
def _built():
    build.build()
    orc.build()
    if native.lib().mcg_device_count() < 1:
        pytest.fail("no CUDA device visible to libmcgpu.so")


def _scale(s):
    t = s.copy()
    t.q = np.abs(t.q)
    e = orc.Oracle(t, moves=False).energy()
    # x^12 - x^6 of a pair is within 4x of x^12 + x^6 wherever it matters here (r above the zero)
    return abs(e[3]) + 4 * abs(e[4]) + sum(abs(v) for v in e[5:10])


def _check(s, got, want):
    scale = _scale(s)
    assert np.all(np.isfinite(got)), got
    assert abs(got[3] - want[3]) <= REL * scale and abs(got[4] - want[4]) <= REL * scale, (got, want, scale)


def _charged_argon(n, seed, **kw):
    s = systems.argon_random(n, 0.0213, seed)
    s.q = np.random.default_rng(seed).normal(0.0, 0.3, n)
    for k, v in kw.items():
        setattr(s, k, v)
    return s


@pytest.mark.parametrize("offset", [0.0, 1e-16, -1e-16, 1e-9, -1e-9, 6e-6, -6e-6, 1.4e-5, -1.4e-5, 1e-4, -1e-4])
@pytest.mark.parametrize("boxes", [0.5, 1.0, 1.5, -1.0, 3.0])
def test_minimum_image_at_its_switch_points(boxes, offset):
    # partners displaced from each other by `boxes` box lengths (times 1 + offset) along each axis in
    # turn, the coordinates left unwrapped as a caller may give them
    # (no Lennard-Jones term: chance overlaps would set the scale)
    s = _charged_argon(48, 5, cut_mode="full")
    s.eps = np.zeros(s.natom)
    L = s.box[0]
    xyz = s.coords()
    for k in range(3):
        i = np.arange(8) + 16 * k
        xyz[i + 8] = xyz[i] + np.array([1.9, 2.3, 3.1])
        xyz[i + 8, k] = xyz[i, k] + L * boxes * (1.0 + offset)
    s.set_coords(xyz)
    got = FFieldCUDA(s, "fp64", moves=False).getE10()
    _check(s, got, np.array(orc.Oracle(s, moves=False).energy()))


def _near(s, seed, jitter=0.3):
    """A configuration with pairs on both sides of the cutoffs: the lattice shaken up."""
    rng = np.random.default_rng(seed)
    s.set_coords(s.coords() + rng.uniform(-jitter, jitter, (s.natom, 3)))
    return s


# 2 atoms (one pair, mostly empty rings), sizes around a block's rows and a ring's 32 pairs, and
# parameter sets on both sides of the class table's limit of 128
@pytest.mark.parametrize("n", [2, 9, 32, 33, 127, 128, 129, 500, 1531])
@pytest.mark.parametrize("box", ["cubic", "orbic"])
def test_switched_energy(n, box):
    s = _near(_charged_argon(n, 11), 12)
    if n < 200:          # boxes of at least the cutoff, so that small systems have pairs at all ranges
        s.box = (25.0, 25.0, 25.0)
        s.set_coords(s.coords() * (25.0 / max(np.ptp(s.coords()), 1.0)) * 0.9)
    if box == "orbic":
        s.pbc_type = "orbic"
        s.box = (s.box[0], s.box[1] * 1.25, s.box[2] * 1.0625)
    got = FFieldCUDA(s, "fp64", moves=False).getE10()
    _check(s, got, np.array(orc.Oracle(s, moves=False).energy()))


# a unit of the full energy is 128 rows by 32 columns; 129 parameter sets leave the class table
@pytest.mark.parametrize("n", [2, 31, 32, 33, 127, 128, 129, 160, 161, 257, 1000])
@pytest.mark.parametrize("box", ["cubic", "orbic"])
def test_full_energy(n, box):
    s = _near(_charged_argon(n, 31, cut_mode="full"), 32)
    if box == "orbic":
        s.pbc_type = "orbic"
        s.box = (s.box[0], s.box[1] * 1.5, s.box[2] * 1.0625)
    got = FFieldCUDA(s, "fp64", moves=False).getE10()
    _check(s, got, np.array(orc.Oracle(s, moves=False).energy()))


def test_full_energy_with_exclusions():
    s = systems.water_box(173, seed=9)
    s.cut_mode = "full"
    got = FFieldCUDA(s, "fp64", moves=False).getE10()
    _check(s, got, np.array(orc.Oracle(s, moves=False).energy()))


# boxes on both sides of twice the pairs' reach (the smallest accepted holds the cutoff sphere exactly)
# The mixed-precision full energy at the edges of its units (128 rows by 32 columns), with and without
# exclusions.  A pair's FP32 r^2 is off by some 6 units of 2^-24 and x^12 takes it to the sixth power:
# 50 such units, 3e-6, with the products behind; the sums are float-float.
@pytest.mark.parametrize("kind,n", [("argon", m) for m in (2, 31, 32, 33, 127, 128, 129, 160, 161, 257, 1000)] +
                         [("water", m) for m in (1, 11, 43, 85, 173)])
@pytest.mark.parametrize("box", ["cubic", "orbic", "none"])
def test_full_energy_mixed(kind, n, box):
    s = _near(_charged_argon(n, 41), 42) if kind == "argon" else systems.water_box(n, seed=43)
    s.cut_mode = "full"
    if box == "orbic":
        s.box = (s.box[0], s.box[1] * 1.5, s.box[2] * 1.0625)
    s.pbc_type = box
    got = FFieldCUDA(s, "mixed", moves=False).getE10()
    want = np.array(orc.Oracle(s, moves=False).energy())
    assert np.all(np.isfinite(got)), got
    tol = 4e-6 * _scale(s)
    assert abs(got[3] - want[3]) <= tol and abs(got[4] - want[4]) <= tol, (got, want, tol)


@pytest.mark.parametrize("L", [24.0, 24.002, 24.003, 25.0])
@pytest.mark.parametrize("box", ["cubic", "orbic"])
def test_switched_energy_smallest_boxes(L, box):
    s = _near(_charged_argon(64, 41), 42)
    s.set_coords(s.coords() * (L / s.box[0]))
    s.box = (L, L, L)
    if box == "orbic":
        s.pbc_type = "orbic"
        s.box = (L, L * 1.25, L * 1.0625)
    got = FFieldCUDA(s, "fp64", moves=False).getE10()
    _check(s, got, np.array(orc.Oracle(s, moves=False).energy()))


@pytest.mark.parametrize("ron", [0.0, 5.0, 11.9])
def test_switched_energy_other_switches(ron):
    s = _near(_charged_argon(600, 3, cuton=ron), 4)
    got = FFieldCUDA(s, "fp64", moves=False).getE10()
    _check(s, got, np.array(orc.Oracle(s, moves=False).energy()))


def _exact_pair(s):
    """(elec, vdw) of atoms 0 and 1 in 60 digits: near the cutoffs the FP64 switch is ill-conditioned."""
    with localcontext() as c:
        c.prec = 60
        D = Decimal
        u = D(0)
        for k, v in enumerate((s.x, s.y, s.z)):
            d, L = D(float(v[1])) - D(float(v[0])), D(float(s.box[k]))
            u += (d - L * (d / L).to_integral_value()) ** 2
        rc2, ron2 = D(s.cutoff) ** 2, D(s.cuton) ** 2
        f = D(0) if u > rc2 else (D(1) if u <= ron2 else (rc2 - u) ** 2 * (rc2 + 2 * u - 3 * ron2) / (rc2 - ron2) ** 3)
        e = [D(float(np.sqrt(v * 418.4))) for v in s.eps[:2]]
        x6 = ((D(float(s.sig[0])) + D(float(s.sig[1]))) ** 2 / u) ** 3
        elec = D(float(332.0716 * 418.4)) * D(float(s.q[0])) * D(float(s.q[1])) / u.sqrt() * f
        return np.array([float(elec), float(4 * e[0] * e[1] * (x6 * x6 - x6) * f)])


# closer than the 64-bit form's limit (some 2e-3 A), at it, above it; on the cutoffs
@pytest.mark.parametrize("r", [1e-5, 1e-3, 2e-3, 4e-3, 0.5, 9.9995, 10.0, 10.0005, 11.9995, 12.0, 12.0005])
def test_one_pair(r):
    s = _charged_argon(3, 7)
    s.box = (40.0, 40.0, 40.0)
    s.set_coords(np.array([[-19.9, 3.0, -2.0], [-19.9 - r * 0.6, 3.0 + r * 0.8, -2.0], [1.0, -12.0, 17.5]]))
    got = FFieldCUDA(s, "fp64", moves=False).getE10()
    want = _exact_pair(s)
    # one term: its displacement carries the coordinates' rounding (2^-49 A) on either side
    rel = 40 * 2.0 ** -53 + 14 * 2.0 ** -48 / r
    assert np.all(np.isfinite(got)) and np.all(np.abs(got[3:5] - want) <= rel * _scale(s) + 1e-30), (got, want)


def test_moves_keep_the_mirror_current():
    s = _near(_charged_argon(700, 21), 22, 0.1)
    ff = FFieldCUDA(s, "fp64", moves=False)
    xyz = s.coords()
    rng = np.random.default_rng(1)
    for _ in range(5):
        idx = rng.choice(s.natom, 3, replace=False)
        new = xyz[idx] + rng.uniform(-0.2, 0.2, (3, 3))
        ff.delta_e(idx, new)
        ff.commit()
        xyz[idx] = new
    got = ff.getE10()
    s.set_coords(xyz)
    o = orc.Oracle(s, moves=False)
    _check(s, got, np.array(o.energy()))


def _check_chains(B, chains):
    e = B.energy_fp64()
    for k in range(0, len(chains), 1 if len(chains) < 8 else 9):
        t = chains[k].copy()
        t.set_coords(B.coords(k))
        want = np.array(orc.Oracle(t, moves=False).energy())
        assert abs(e[k] - (want[3] + want[4])) <= REL * _scale(t), (k, e[k], want)


# tiles of 8 residues, of 32 (one-atom residues from 19,456 in all) and of 16 (others from 155,648), residue sizes 1
# and 3 and both
@pytest.mark.parametrize("sizes", [[("water", 513)], [("argon", 331), ("argon", 513)], [("water", 512), ("argon", 640), ("water", 519)],
                                   [("water", 6500), ("water", 6489), ("water", 6511)],
                                   [("argon", 2001 + k) for k in range(10)], [("water", 8177 + k) for k in range(20)]])
def test_batch_energy(sizes):
    chains = [systems.water_box(n, seed=n) if kind == "water" else systems.argon_random(n, 0.0213, n) for kind, n in sizes]
    if len(chains) == 2:
        chains[1].pbc_type = "orbic"
        chains[1].box = (chains[1].box[0], chains[1].box[1] * 1.25, chains[1].box[2] * 1.0625)
    B = BatchChains(chains, seed=3)
    _check_chains(B, chains)
    B.sweep(1)
    _check_chains(B, chains)


# The mixed recompute over residue lists: rows that start at an odd entry, lists of no entry to some 30
# (dilute chains) and of hundreds, residue sizes 1 and 3 and both.  The pair terms' error is as in
# test_full_energy_mixed; the switch polynomial's few units come on top of its 50.
@pytest.mark.parametrize("kinds", [["argon"], ["water"], ["argon", "water"]])
@pytest.mark.parametrize("cap", [0, 1023])
def test_batch_energy_mixed_lists(kinds, cap):
    chains = []
    for kind in kinds:
        for n, density in ((90, 2e-4), (200, 2e-3), (700, 0.0213)) if kind == "argon" else ((517, 0.0), (600, 0.0)):
            chains.append(systems.argon_random(n, density, n) if kind == "argon" else systems.water_box(n, seed=n))
    B = BatchChains(chains, seed=3, list_capacity=cap)
    got, want = B.energy_mixed(), B.energy_fp64()
    for k, s in enumerate(chains):
        assert abs(got[k] - want[k]) <= 4e-6 * _scale(s), (k, got[k], want[k])


def test_batch_energy_of_residues_wider_than_at_creation():
    chains = [systems.water_box(600, seed=1)]
    B = BatchChains(chains, seed=3)
    xyz = chains[0].coords()
    xyz[4] += [4.0, -5.0, 6.0]
    xyz[901] += [-9.0, 0.0, 2.0]
    B.set_coords(0, xyz)
    _check_chains(B, chains)


# row-build tasks of 2 and 4 home atoms (4 from 8,192 atoms), cells with a few and many atoms, few cells
# an axis (whole-axis stencils) and many, an orthorhombic box, and no box at all
@pytest.mark.parametrize("kind,n", [("argon", 331), ("argon", 9001), ("water", 700), ("water", 2730), ("water", 2731), ("orbic", 5003),
                                    ("vacuum", 3001)])
def test_verlet_rows(kind, n):
    s = systems.water_box(n, seed=n) if kind == "water" else _near(_charged_argon(n, n), 1)
    if kind == "orbic":
        s.pbc_type = "orbic"
        s.box = (s.box[0], s.box[1] * 1.5, s.box[2] * 1.0625)
    if kind == "vacuum":
        s.pbc_type = "none"
    s.frozen = (np.arange(s.natom) % 3 == 0).astype(np.uint8) if n % 2 else s.frozen
    rows = FFieldCUDA(s, "fp64", moves=False).pairlist()
    want = orc.Oracle(s, moves=False).verlet_rows()
    assert all(np.array_equal(a, np.sort(b)) for a, b in zip(rows, want, strict=True))


# builds after each other on one handle, without a box: the cell grid grows and shrinks between them and
# the rows outgrow their capacity; the counters that one build leaves behind are the next one's
def test_verlet_rows_of_successive_builds():
    s = _near(_charged_argon(1200, 17), 18)
    s.pbc_type = "none"
    xyz = s.coords()
    ff = FFieldCUDA(s, "fp64", moves=False)
    for scale in (1.0, 1.9, 0.6, 1.2, 1.2):
        s.set_coords(xyz * scale)
        ff.setCoords(s.coords())
        ff.askListUpdate(0)
        want = orc.Oracle(s, moves=False).verlet_rows()
        assert all(np.array_equal(a, np.sort(b)) for a, b in zip(ff.pairlist(), want, strict=True))


def _bonded_chain(n, seed, angles, torsion_kinds):
    """n charged atoms in a chain whose angles and torsions take the given values (degrees), with terms
    referred to other values: from no deviation to the whole circle."""
    s = systems.argon_random(n, 0.005, seed)
    rng = np.random.default_rng(seed)
    xyz = [np.zeros(3), np.array([1.5, 0.0, 0.0])]
    for i in range(2, n):
        th, ph = np.radians(angles[i % len(angles)]), rng.uniform(-np.pi, np.pi)
        u = xyz[-1] - xyz[-2]
        u /= np.linalg.norm(u)
        v = np.cross(u, [0.3, 0.5, 0.81])
        v /= np.linalg.norm(v)
        w = np.cross(u, v)
        xyz.append(xyz[-1] + 1.5 * (-np.cos(th) * u + np.sin(th) * (np.cos(ph) * v + np.sin(ph) * w)))
    s.set_coords(np.array(xyz))
    s.pbc_type, s.cut_mode = "none", "full"
    s.eps = np.zeros(n)
    s.angles = np.stack([np.arange(n - 2), np.arange(1, n - 1), np.arange(2, n)], 1).astype(np.int32)
    s.angle_type = np.zeros(n - 2, np.int32)
    s.angle_k = np.full(n - 2, 55.0)
    s.angle_theta0 = np.array([angles[i % len(angles)] + d for i, d in zip(range(2, n), np.tile([0.0, 1e-9, 0.3, 0.8, 0.95, 5.0, -40.0], n))])
    d4 = np.stack([np.arange(n - 3), np.arange(1, n - 2), np.arange(2, n - 1), np.arange(3, n)], 1).astype(np.int32)
    m = n - 3
    s.dihedrals, s.dihe_type = d4, np.array([torsion_kinds[k % len(torsion_kinds)][0] for k in range(m)], np.int32)
    s.dihe_mult = np.array([torsion_kinds[k % len(torsion_kinds)][1] for k in range(m)], np.float64)
    s.dihe_order = np.maximum(1, s.dihe_mult).astype(np.int32)
    s.dihe_k, s.dihe_phi0 = rng.uniform(0.1, 2.0, m), rng.uniform(-180, 180, m)
    s.impropers, s.impr_type = d4.copy(), np.full(m, 2, np.int32)
    s.impr_order, s.impr_mult, s.impr_k = np.ones(m, np.int32), np.ones(m), np.full(m, 20.0)
    a, b, c, d = (s.coords()[d4[:, k]] for k in range(4))
    n1, n2 = np.cross(a - b, b - c), np.cross(b - c, c - d)
    phi = np.degrees(np.arctan2((np.cross(n2, n1) * (b - c)).sum(1) / np.linalg.norm(b - c, axis=1), (n1 * n2).sum(1)))
    s.impr_phi0 = phi + np.tile([0.0, 1e-9, 0.5, 0.89, 0.91, 60.0, 180.0, 359.7], n)[:m]
    return s


# angles from a right one to nearly straight, multiplicities that are and are not small integers, harmonic
# torsions from their reference value to half a turn off it
@pytest.mark.parametrize("angles", [[90.0, 104.52, 111.0], [3.0, 30.0, 150.0], [176.0, 177.6, 179.9]])
@pytest.mark.parametrize("kinds", [[(1, 1), (1, 2), (1, 3)], [(1, 0), (1, 6), (1, 7), (1, 2.5)], [(2, 1), (1, 1)]])
def test_bonded_terms(angles, kinds):
    s = _bonded_chain(60, 8, angles, kinds)
    got = FFieldCUDA(s, "fp64", moves=False).getE10()
    want = np.array(orc.Oracle(s, moves=False).energy())
    # an angle or torsion near its ends magnifies a coordinate's rounding by 1 / sin(theta) and the torsion
    # by that of both its angles; a term's error is that times its slope, k |deviation|
    amp = 1.0 / np.sin(np.radians(min(min(angles), 180 - max(angles)))) ** 2
    dev = 2.0 ** -49 * amp * 8
    slope = KCAL * (55.0 * np.radians(45) + 2.0 * 7) * s.natom, KCAL * 20.0 * np.pi * s.natom
    assert abs(got[6] - want[6]) <= dev * slope[0], (got, want)
    assert abs(got[8] - want[8]) <= dev * (slope[0] + slope[1]) and abs(got[9] - want[9]) <= dev * slope[1], (got, want)


# proposals inside the launch (up to 32 atoms and 192 bonded terms) and staged beside it, one block per bonded
# kind, every precision and cutoff; mixed precision to the engine's own 1e-4 kcal/mol per trial move of a
# residue of three atoms, independent errors of more atoms adding in quadrature
@pytest.mark.parametrize("prec,cut", [("fp64", "switch"), ("fp64", "full"), ("mixed", "switch")])
@pytest.mark.parametrize("m", [1, 3, 31, 32, 33, 40, 200])
def test_trial_moves(prec, cut, m):
    s = systems.peptide_in_water(40, 700, L=30.0, seed=6)
    s.cut_mode = cut
    ff = FFieldCUDA(s, prec, moves=False)
    o = orc.Oracle(s, moves=False)
    e0 = np.array(o.energy())
    rng = np.random.default_rng(m)
    idx = np.sort(rng.choice(40 if m <= 40 else s.natom, m, replace=False))
    new = s.coords()[idx] + rng.uniform(-0.02, 0.02, (m, 3))
    de = ff.delta_e(idx, new)
    xyz = s.coords()
    xyz[idx] = new
    o.set_coords(xyz)
    want = np.array(o.energy())[0] - e0[0]
    # the oracle's own difference of two totals carries both sums' rounding
    tol = 1e-4 * KCAL * max(1.0, (m / 3) ** 0.5) if prec == "mixed" else 2 * REL * _scale(s)
    assert abs(de - want) <= tol, (de, want, tol)


# moves of several atoms in the device-resident run: pairs inside the moved set, terms of one atom's row on
# other threads than the next's, and the order of the commits
@pytest.mark.parametrize("apr", [1, 2, 3, 7, 64])
def test_device_run_moves_of_several_atoms(apr):
    s = systems.argon_fcc(6)
    s.resid = np.arange(s.natom, dtype=np.int32) // apr + 1
    s.moves[0].move_mode = "residue"
    dev, host = FFieldCUDA(s, "fp64"), FFieldCUDA(s, "fp64")
    l0 = dev.kernel_launches()
    _, e_dev, a_dev, _ = dev.metropolis(400, 7, acceptance="physical", trace=False)
    assert dev.kernel_launches() - l0 < 200          # on the device: a launch per 50 steps and the list builds
    _, e_host, a_host, _ = host.metropolis(400, 7, acceptance="physical", trace=True)
    assert a_dev == a_host and np.array_equal(dev.coords(), host.coords())
    assert abs(e_dev - e_host) <= 1e-10 * abs(e_host)


def test_coordinates_that_are_refused_leave_the_engine_as_it_was():
    s = _near(_charged_argon(2500, 5), 6)
    ff = FFieldCUDA(s, "fp64", moves=False)
    e = ff.getE10()
    for at, v in ((0, np.nan), (1024, np.inf), (2499, -np.inf)):
        bad = s.coords() + 0.01
        bad[at, at % 3] = v
        with pytest.raises(native.McgError, match="atom %d" % at):
            ff.setCoords(bad)
        assert np.array_equal(ff.coords(), s.coords()) and np.array_equal(ff.getE10(), e)
        assert ff.getE_host(s.x, s.y, s.z) == e[0]
