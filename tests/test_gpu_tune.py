"""Tuned engines give the results of untuned ones: every CTA size of the batched base-2 launch, and
the sieve, the Fermat quotients and BPSW after the autotuner's choice."""
import numpy as np
import pytest

import mathpub_b200 as mp

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng():
    e = mp.Engine(0)
    yield e
    e.close()


@pytest.mark.parametrize("variant", [0, 1, 2, 3])
@pytest.mark.parametrize("count", [8193, 60001])
def test_bpsw_cta_sizes(eng, variant, count):
    n, _ = mp.bpsw_workload(17, count, 1)
    with mp.Engine(0) as other:
        want = other.bpsw(n)
    eng.tune_set(bpsw_variant=variant)
    assert np.array_equal(eng.bpsw(n), want)


def test_results_after_autotune(eng):
    lo, hi = 10 ** 12 + 1, 10 ** 12 + 2 ** 27 + 77
    with mp.Engine(0) as other:
        want = other.sieve_range(lo, hi, block_log2=24, hash_log2=20)
        p = other.primes_range(lo, lo + 10 ** 6)
        q, prime = other.fermat_quotient(p), other.bpsw(np.arange(lo, lo + 20000, dtype=np.uint64))
    report = eng.autotune(10 ** 15)
    assert [s for s in report.splitlines() if s.startswith("sieve choice:")]
    got = eng.sieve_range(lo, hi, block_log2=24, hash_log2=20)
    for k in want:
        assert np.array_equal(np.asarray(got[k]), np.asarray(want[k])), k
    assert np.array_equal(eng.fermat_quotient(p), q)
    assert np.array_equal(eng.bpsw(np.arange(lo, lo + 20000, dtype=np.uint64)), prime)
