"""Every CTA size of the batched base-2 launch against the oracle, on more candidates than the one-launch form
takes (16,384): the first count above it, and ones whose last CTAs are partly filled."""
import numpy as np
import pytest

import mathpub_b200 as mp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant", [0, 1, 2, 3])
def test_batched(orc, variant):
    n, _ = mp.bpsw_workload(17, 100003, 1)
    want = orc.bpsw(n)
    with mp.Engine(0) as e:
        e.tune_set(bpsw_variant=variant)
        for count in (16385, 16417, 60001, 100003):
            assert np.array_equal(e.bpsw(n[:count]), want[:count]), count
            assert np.array_equal(e.bpsw(n[-count:]), want[-count:]), count
