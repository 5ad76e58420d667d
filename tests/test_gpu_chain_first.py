"""chain_first over ranges far longer than the stretch that holds the first chain: the first chain of the long
range is the first of a short one, also where it lies past the part that the short ranges' plan takes, and the
call costs about as much as the same search in a range of 1e12 integers."""
import time

import pytest

import mathpub_b200 as mp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dec", [False, True])
@pytest.mark.parametrize("k", [4, 5, 6, 8, 10])
def test_long_range(engine, k, dec):
    lo = 10 ** 16 + 3
    n = 10 ** 13 if k == 10 else 10 ** 12
    assert engine.chain_first(lo, 2 ** 63, k, dec=dec) == engine.chain_first(lo, lo + n, k, dec=dec)


@pytest.mark.parametrize("dec", [False, True])
def test_past_the_near_part(engine, dec):
    """The first chain of 12 from 1.3e17 on, searched from far and from near below it."""
    lo, hi, k = 13 * 10 ** 16, 13 * 10 ** 16 + 4 * 10 ** 15, 12
    got = engine.chain_first(lo, hi, k, dec=dec)
    h, l = engine.chain_sieve(lo, hi, k, dec=dec)
    if got is None:
        assert len(h) == 0
    else:
        assert got[1] == int(h[0]) and got[2] == int(l[0])
        assert engine.chain_first(got[0], got[0] + 10 ** 6, k, dec=dec) == got
        assert engine.chain_first(got[0] - 110 * 10 ** 12, hi, k, dec=dec) == engine.chain_first(
            got[0] - 110 * 10 ** 12, got[0] + 1, k, dec=dec)


def test_cost_of_a_long_range():
    """The first chain of 4 lies within 1e6 integers: a search to 2^63 takes no more than four times one over 1e12
    integers (20 times, when the range's length chose the wheel)."""
    with mp.Engine(0) as e:
        def best(hi):
            t = []
            for _ in range(5):
                a = time.perf_counter()
                e.chain_first(10 ** 16, hi, 4)
                t.append(time.perf_counter() - a)
            return min(t)
        assert best(2 ** 63) < 4 * best(10 ** 16 + 10 ** 12)
