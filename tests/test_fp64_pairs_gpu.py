"""FP64 pair arithmetic and energy kernels where they can go wrong, against the FP64 oracle.

Tolerance: a pair term carries at most about 40 roundings on either side (twelve of them through
x^12), and a sum of N terms as many as its longest chain of additions, so 1e-13 of the sum of the
terms' magnitudes bounds both for the sizes here.  Only totals are visible, so the magnitude is
taken from the oracle's energies of the attractive and repulsive parts, |elec| + |vdw| of the same
system with all charges made positive.
"""
import numpy as np
import pytest

import oracle as orc
from mc_cpp_gb300 import build, native, systems
from mc_cpp_gb300.engine import FFieldCUDA

pytestmark = pytest.mark.gpu
REL = 1e-13


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
