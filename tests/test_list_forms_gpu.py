"""Verlet rows of the list build's other forms, as sets against the FP64 oracle's: systems with frozen atoms
(a flag per home atom and candidate).
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
