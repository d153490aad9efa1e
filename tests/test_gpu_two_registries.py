"""A registry keeps working when another one, set up for fewer slots and tiles, is created beside it: the shared memory that a kernel may take is
the kernel's, not the registry's."""
import numpy as np
import pytest

import harness

pytestmark = pytest.mark.gpu


def test_a_smaller_registry_beside_a_larger_one(pe):
    from pocket_engine_b200 import workloads
    site = pe.Site.fused(0, 256, [("a", 128)])
    wl = workloads.Workload("beside", [site], [16], 1.0, [1, 3], [1, 1], 5)
    large = harness.product_registry(pe, wl, max_slots=500)  # over the 48 KB that a launch may take by default
    before = harness.run_gpu(pe, large, wl, True)
    small = harness.product_registry(pe, wl, max_slots=2)
    after = harness.run_gpu(pe, large, wl, True)
    assert np.array_equal(before[0], after[0])
    small.close()
    large.close()
