"""The one-launch form for few candidates against the oracle at the limits of its two sizes and of a
CTA, on values of every phase: small and even numbers, squares, strong base-2 and strong Lucas
pseudoprimes, both size classes of the base-2 test, and 2^64 - 1."""
import numpy as np
import pytest

import mathpub_b200 as mp

pytestmark = pytest.mark.gpu


def values(ref_vectors):
    rng = np.random.default_rng(11)
    xs = list(range(0, 300)) + list(range(17000, 17400))
    xs += [1093 ** 2, 3511 ** 2, 131 ** 2, 65537 ** 2, (2 ** 32 - 5) ** 2, 2 ** 64 - 1, 2 ** 64 - 59, 2 ** 63 - 25, 2 ** 63 + 29]
    xs += [int(r) ** 2 for r in rng.integers(2 ** 20, 2 ** 32, 60)]
    xs += list(ref_vectors["spsp2"])[:300] + list(ref_vectors["slpsp"])[:300]
    xs += [2 ** 64 - 1 - 2 * k for k in range(1, 300)] + [2 ** 63 + k for k in range(-199, 200, 2)]
    n, _ = mp.bpsw_workload(5, 16385 - len(xs), 1)
    return rng.permutation(np.concatenate([np.array(xs, dtype=np.uint64), n]))


@pytest.mark.parametrize("count", [1, 7, 8, 9, 31, 32, 33, 2016, 2017, 2048, 2049, 16352, 16384, 16385])
def test_counts(engine, orc, ref_vectors, count):
    n = values(ref_vectors)
    for part in (n[:count], n[-count:]):
        assert np.array_equal(engine.bpsw(part), orc.bpsw(part))
