"""Verlet rows of the list build's other forms, as sets against the FP64 oracle's: systems without a box (FP32
coordinates place most pairs, up to an extent of 20 list radii; beyond it the FP64 test takes all), frozen atoms
(a flag per home atom), and cells of hundreds of atoms (512 threads a cell, more than 2,048 unsorted in shared
memory).  Partners are put within 1e-9 to 1e-3 of the list radius, on both sides, where FP32 may not decide.
"""
import numpy as np
import pytest

import oracle as orc
from mc_cpp_gb300 import build, native, systems
from mc_cpp_gb300.engine import FFieldCUDA

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    build.build()
    orc.build()
    if native.lib().mcg_device_count() < 1:
        pytest.fail("no CUDA device visible to libmcgpu.so")


def _compare(s):
    rows = FFieldCUDA(s, "fp64", moves=False).pairlist()
    want = orc.Oracle(s, moves=False).verlet_rows()
    assert all(np.array_equal(a, np.sort(b)) for a, b in zip(rows, want, strict=True))
    return sum(len(r) for r in rows)


def _atoms(n, extent, seed):
    """n atoms over a cube of the given extent, a third of them partners of others at about the list radius."""
    s = systems.argon_random(n, 0.0213, seed)
    rng = np.random.default_rng(seed)
    xyz = rng.uniform(0.0, extent, (n, 3))
    k = n // 3
    v = rng.normal(size=(k, 3))
    r = 14.0 * (1.0 + rng.choice([-1.0, 1.0], k) * 10.0 ** rng.uniform(-9, -3, k))
    xyz[n - k:] = xyz[:k] + v * (r / np.linalg.norm(v, axis=1))[:, None]
    s.set_coords(xyz)
    s.pbc_type = "none"
    return s


# 20 list radii are 280 A
@pytest.mark.parametrize("extent", [5.0, 60.0, 240.0, 300.0, 2e4])
@pytest.mark.parametrize("offset", [0.0, -1e5])
@pytest.mark.parametrize("n", [2, 45, 1500])
def test_rows_without_a_box(n, extent, offset):
    s = _atoms(n, extent, n)
    s.set_coords(s.coords() + offset)
    _compare(s)


@pytest.mark.parametrize("n", [8191, 8192])
def test_rows_without_a_box_at_the_task_size(n):
    assert _compare(_atoms(n, 90.0, n)) > 100000


@pytest.mark.parametrize("kind", ["cubic", "none"])
@pytest.mark.parametrize("frozen", ["one", "third", "all but one", "all"])
@pytest.mark.parametrize("nmol", [600, 2800])
def test_rows_with_frozen_atoms(kind, frozen, nmol):
    s = systems.water_box(nmol, seed=nmol)
    s.pbc_type = kind
    n = s.natom
    s.frozen = {"one": np.arange(n) == 7, "third": np.random.default_rng(1).random(n) < 0.33,
                "all but one": np.arange(n) != 7, "all": np.ones(n, bool)}[frozen].astype(np.uint8)
    total = _compare(s)
    assert (total == 0) == (frozen == "all")


@pytest.mark.parametrize("n", [255, 256, 2047, 2049, 2500])
@pytest.mark.parametrize("kind", ["cubic", "none"])
def test_rows_of_crowded_cells(n, kind):
    s = systems.argon_random(n, 0.0213 * 125, n)       # one cell: the box is at most 10 A, the list radius more than half
    s.cutoff, s.cuton, s.sig = s.box[0] / 2.1, s.box[0] / 4, s.sig / 5
    s.pbc_type = kind
    _compare(s)


# rows that would need more memory than any device has: the update fails, what needs rows is refused until an
# update succeeds, and then everything is as before.  (Two million atoms drawn together to 45,000 partners each
# would take 400 GB; their 1,400 to a cell stay within a cell's sort.)
def test_rows_that_do_not_fit_the_device():
    n = 2_000_000
    s = systems.argon_random(n, n / 300.0 ** 3, 5)
    ff = FFieldCUDA(s, "fp64", moves=False)
    e = ff.getE10()
    idx, new = np.array([3], np.int32), s.coords()[3:4] + 0.01
    de = ff.delta_e(idx, new)
    ff.setCoords(np.random.default_rng(6).uniform(0.0, 80.0, (n, 3)))
    with pytest.raises(native.McgError, match="cudaMalloc"):
        ff.askListUpdate(0)
    for call in (ff.getE10, lambda: ff.delta_e(idx, new), lambda: ff.time_nonbonded(1)):
        with pytest.raises(native.McgError, match="no Verlet list"):
            call()
    ff.setCoords(s.coords())
    ff.askListUpdate(0)
    assert np.array_equal(ff.getE10(), e) and ff.delta_e(idx, new) == de
