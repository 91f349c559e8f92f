"""Group rows at the ends of the bitmap build's range (one-atom groups, so atoms are groups): a bitmap's
words come in runs of 1,024 groups, and above 65,536 groups the hash table builds the rows.  Every pair
of the source rows has to be one mask bit, and the group kernel has to give the list kernel's energy to the
FP32 summation order (2e-7 of its terms)."""
from concurrent.futures import ThreadPoolExecutor

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


@pytest.mark.parametrize("n", [400, 1023, 1024, 1025, 65535, 65536, 65537])
def test_rows_around_the_limits(n):
    s = systems.argon_random(n, 0.0213, n)
    ff = FFieldCUDA(s, "mixed", moves=False)
    groups, entries, bits = ff.group_stats()
    assert groups == n and entries == bits == ff.prune_stats()[0]
    ff.set_pair_kernel(0)
    want = ff.getE10()
    ff.set_pair_kernel(7)
    got = ff.getE10()
    assert abs(got[4] - want[4]) <= 2e-7 * abs(want[4]) and np.all(np.isfinite(got))


# handles of different sizes whose rows are built in several threads at once: the bitmap kernel's limit of
# shared memory belongs to the process (72 and 96 KB here), and a build must not lower it under another's launch
def test_rows_built_in_several_threads():
    ffs = [FFieldCUDA(systems.argon_random(n, 0.0213, n), "mixed", moves=False) for n in (46000, 65000, 46500, 64000)]
    want = [ff.group_stats() for ff in ffs]
    assert all(w[1] > 0 for w in want)

    def build_rows(k):
        for _ in range(600):
            ffs[k].askListUpdate(0)
            if ffs[k].group_stats() != want[k]:
                return False
        return True
    with ThreadPoolExecutor(len(ffs)) as pool:
        assert all(pool.map(build_rows, range(len(ffs))))
