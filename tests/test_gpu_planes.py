"""The residue-plane sieve (the batched default) against the oracle where its parts meet: ranges of one
tile and of several waves' worth of tiles, starts below the first sieving primes and at every residue
mod 30, block sizes at the edge of the scan's stretches, heights where every large prime is a bucket
prime, and prime lists against the same ranges' counts and bitmaps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KEYS = ("pi", "twins", "max_gap", "gap_start", "tuple6", "tuple6_cks", "first_prime", "last_prime")


def check(engine, orc, lo, hi, **kw):
    r, o = engine.sieve_range(lo, hi, **kw), orc.sieve_range(lo, hi, **kw)
    assert {k: r[k] for k in KEYS} == {k: int(o[k]) for k in KEYS}, (lo, hi)
    for k in ("blocks", "hashes", "bitmap"):
        if k in r:
            assert np.array_equal(r[k], o[k]), (k, lo, hi)


@pytest.mark.parametrize("lo", list(range(0, 34)) + [88, 89, 90, 96, 97, 2999, 30 * 10 ** 11 + 7, 2 ** 64 - 2 ** 24])
def test_starts(engine, orc, lo):
    for n in (1, 7, 30, 961, 70000, 2 ** 20 + 5):
        hi = min(lo + n, 2 ** 64 - 2 ** 18)
        check(engine, orc, lo, hi, bitmap=True, hash_log2=12)


@pytest.mark.parametrize("lo,n,block_log2", [
    (10 ** 9 + 7, 5 * 2 ** 22 + 12345, 21), (10 ** 9, 2 ** 26 - 2, 24), (10 ** 12 + 1, 2 ** 27 + 31, 22),
    (3 * 10 ** 14, 2 ** 28, 26), (10 ** 16, 2 ** 24 + 1, 21), (5 * 10 ** 18, 2 ** 25 - 17, 23)])
def test_blocks(engine, orc, lo, n, block_log2):
    check(engine, orc, lo, lo + n, block_log2=block_log2, hash_log2=19)


@pytest.mark.parametrize("lo,n", [(10 ** 9, 2 ** 33 + 2 ** 30 + 99), (10 ** 15 + 11, 2 ** 32 + 7), (9 * 10 ** 17, 2 ** 31)])
def test_long_equals_odd_only_tiles(engine, lo, n):
    """Several waves and the largest tiles, against the odd-only form."""
    a = engine.sieve_range(lo, lo + n, block_log2=26, hash_log2=24)
    b = engine.sieve_range(lo, lo + n, block_log2=26, hash_log2=24, tile_log2=20)
    assert all(a[k] == b[k] for k in KEYS)
    assert np.array_equal(a["blocks"], b["blocks"]) and np.array_equal(a["hashes"], b["hashes"])


@pytest.mark.parametrize("lo,n", [(0, 1000), (1, 100000), (4, 30), (10 ** 9, 123), (10 ** 12 + 17, 2 ** 22 + 3),
                                  (10 ** 15, 3 * 10 ** 7), (10 ** 18, 2 ** 21)])
def test_prime_lists(engine, orc, lo, n):
    p = engine.primes_range(lo, lo + n)
    assert np.array_equal(p, orc.primes_range(lo, lo + n))
