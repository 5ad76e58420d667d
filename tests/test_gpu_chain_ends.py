"""The constellation sieve's last values of k: counts of sextuplets and chains of ranges that end around a whole
number of wheels (a chunk's, a word's and a segment's first and last k, for the classes on both sides of the end)
against a longer range less its rest, which has other offsets; short ranges against the oracle."""
import pytest

pytestmark = pytest.mark.gpu

SEXT = (0, 4, 6, 10, 12, 16)
W = 9699690                                     # the wheel of the primes up to 19
M = 2 ** 64


@pytest.mark.parametrize("lo", [10 ** 15, 3 * 10 ** 12 + 4849845])
def test_ends(engine, lo):
    top = lo + W * 140000
    n, c = engine.tuple_count(lo, top, SEXT)
    for m in (1, 31, 32, 33, 127, 128, 129, 4096, 131071, 131072, 131073):
        for d in (-1, 0, 1, W // 2):
            hi = lo + W * m + d
            a, b = engine.tuple_count(lo, hi, SEXT), engine.tuple_count(hi, top, SEXT)
            assert (a[0] + b[0], (a[1] + b[1]) % M) == (n, c), (m, d)


@pytest.mark.parametrize("lo,k", [(10 ** 12, 5), (10 ** 15, 6)])
def test_short_ranges(engine, orc, lo, k):
    for n in (1, 2, 1000, W - 1, W, W + 1, 33 * W + 17):
        h, l = engine.chain_sieve(lo, lo + n, k)
        want = orc.gap_chains(lo, lo + n, k)
        assert list(zip(h.tolist(), l.tolist())) == sorted((int(x), int(y)) for x, y in zip(*want)), n
