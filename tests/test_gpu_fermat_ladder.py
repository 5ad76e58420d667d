"""The windowed negative-exponent ladder of the Fermat-quotient kernels against Python's integers:
the smallest moduli (no squaring at all), every length of the exponent's first window, digits at
both ends, the limits of the three- and four-limb forms, and composites (pseudoprimes to base 2
have a quotient; for any other composite the result is the one the definition gives on 64 bits)."""
import numpy as np
import pytest

import mathpub_b200 as mp

pytestmark = pytest.mark.gpu

NO_QUOTIENT = 2 ** 64 - 1


def want(p):
    if p < 3 or p % 2 == 0:
        return 0
    q = (pow(2, p - 1, p * p) - 1) * pow(p, -1, 2 ** 64) % 2 ** 64
    return q if q < p else NO_QUOTIENT


@pytest.fixture(scope="module")
def engine():
    e = mp.Engine(0)
    yield e
    e.close()


@pytest.mark.parametrize("limit", [2 ** 47, 2 ** 63])
def test_edges(engine, limit):
    ps = list(range(0, 700)) + [1093, 3511, 341, 561, 2047, 1194649, 12327121]
    for b in range(6, limit.bit_length()):
        ps += [(1 << b) + o for o in (-3, -1, 1, 3, 5, 7)]
        ps += [((1 << b) // 31 | 1) + o for o in (-2, 0, 2)]              # digits of 1 and of 32
    ps += [limit - o for o in range(1, 120, 2)]
    ps = np.array([p for p in ps if 0 <= p < limit], dtype=np.uint64)
    got = engine.fermat_quotient(ps)
    for p, q in zip(ps.tolist(), got.tolist()):
        assert q == want(p), p


@pytest.mark.parametrize("bits", [33, 41, 46, 47, 48, 54, 62, 63])
def test_random_odd(engine, bits):
    r = np.random.default_rng(bits)
    ps = r.integers(1 << (bits - 1), 1 << bits, 2000, dtype=np.uint64) | np.uint64(1)
    got = engine.fermat_quotient(ps)
    assert got.tolist() == [want(p) for p in ps.tolist()]


def test_two_primes_per_thread(engine):
    ps = np.arange(3, 4004, 2, dtype=np.uint64) + np.uint64(10 ** 12)
    a = engine.fermat_quotient(ps)
    engine.tune_set(fermat_ilp2=1)
    b = engine.fermat_quotient(ps)
    engine.tune_set(fermat_ilp2=0)
    assert np.array_equal(a, b)
