"""The device-resident Metropolis run with move-instance tables on both sides of its staging memory (some 43,000
one-atom instances), against the host loop: the same moves, decisions and coordinates."""
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


@pytest.mark.parametrize("n", [3000, 43000, 43600, 60000])
def test_tables(n):
    s = systems.argon_random(n, 0.0213, 9)
    dev, host = FFieldCUDA(s, "fp64"), FFieldCUDA(s, "fp64")
    l0 = dev.kernel_launches()
    _, e_dev, a_dev, _ = dev.metropolis(120, 5, acceptance="physical", trace=False)
    assert dev.kernel_launches() - l0 < 60       # on the device: a launch per 50 steps and the list builds
    _, e_host, a_host, _ = host.metropolis(120, 5, acceptance="physical", trace=True)
    assert 0 < a_dev < 120 and a_dev == a_host and np.array_equal(dev.coords(), host.coords())
    assert abs(e_dev - e_host) <= 1e-10 * abs(e_host)
    # what follows the run reads its mirrors: an energy, and the energy of the same coordinates on a new handle
    t = s.copy()
    t.set_coords(dev.coords())
    dev.askListUpdate(0)
    assert np.array_equal(dev.getE10(), FFieldCUDA(t, "fp64", moves=False).getE10())
