"""The mixed full energy's sums: a pair's FP32 Lennard-Jones term is the same bit for bit whichever atom comes
first (differences of box fractions change sign exactly, sigma sums and eps products commute), so the order of the
atoms changes the total only by how the terms are summed.  Thousands of pairs of a thread are float-float over
short runs (48 bits of a run's largest sum, runs independent of one another) and FP64 beyond, which leaves a
few units in the last place of the total: 4 are allowed.
"""
import numpy as np
import pytest

from mc_cpp_gb300 import build, native, systems
from mc_cpp_gb300.engine import FFieldCUDA

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    build.build()
    if native.lib().mcg_device_count() < 1:
        pytest.fail("no CUDA device visible to libmcgpu.so")


@pytest.mark.parametrize("n", [4096, 36864])
def test_order_of_atoms(n):
    s = systems.argon_random(n, 0.0213, 3)
    s.cut_mode = "full"
    want = FFieldCUDA(s, "mixed", moves=False).getE10()[4]
    for k in range(3):
        t = s.copy()
        t.set_coords(s.coords()[np.random.default_rng(k + 1).permutation(n)])
        assert abs(FFieldCUDA(t, "mixed", moves=False).getE10()[4] - want) <= 4 * 2.0 ** -52 * abs(want)
