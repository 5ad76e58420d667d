"""Two equally wide gaps in a range: gap_start is the prime before the first of them, in the range's result,
the blocks' and a served request's.  The earlier gap goes from 1 to 29 mod 30 and so holds one block of 30
without a prime fewer than the later one: 58 (none against one), 88, 148 and 268 (1, 3 and 7 against one
more), with both gaps within the 1024 blocks that the scan takes at a time.  Batched against the oracle, the
odd-only tiles and the plain form."""
import numpy as np
import pytest

import mathpub_b200 as mp

pytestmark = pytest.mark.gpu

TIES = [
    (58, 58829, 79758), (58, 1043219, 1043833), (58, 7272059, 7273903), (58, 1000000159619, 1000000159753),
    (88, 5268809, 5274553), (88, 7052609, 7062289), (88, 29146799, 29164339),
    (148, 223125869, 223146169), (148, 818768609, 818776699), (148, 837162959, 837188833),
    (148, 1019880000, 1019900000), (148, 1000097280000, 1000097300000),
    (268, 1000005102882359, 1000005102895063), (268, 1000005132740159, 1000005132745039),
    (268, 1000005796281239, 1000005796308259),
]


@pytest.mark.parametrize("gap,lo,hi", TIES)
def test_first_of_two(engine, orc, gap, lo, hi):
    want = orc.sieve_range(lo, hi)
    assert int(want["max_gap"]) == gap
    start = int(want["gap_start"])
    for kw in ({}, {"tile_log2": 18}, {"mode": mp.MODE_PLAIN}):
        r = engine.sieve_range(lo, hi, **kw)
        assert (r["max_gap"], r["gap_start"]) == (gap, start), kw
    # the same two gaps elsewhere in a stretch of the scan
    for back in (1, 30, 961, 4000):
        a, b = engine.sieve_range(lo - back, hi, bitmap=True), orc.sieve_range(lo - back, hi)
        assert (a["max_gap"], a["gap_start"]) == (int(b["max_gap"]), int(b["gap_start"])), back


def test_blocks(engine, orc):
    """Blocks that begin at the earlier gap's prime."""
    for gap, lo, hi in TIES:
        if hi - lo > 2 ** 15:
            continue
        a, b = (x.sieve_range(lo, lo + 2 ** 21, block_log2=21) for x in (engine, orc))
        assert np.array_equal(a["blocks"], b["blocks"]), (gap, lo)


def test_every_window(engine, orc):
    """Many windows of 20,000 integers, where a warp of the scan has one row."""
    lo = 10 ** 6
    p = orc.primes_range(lo, lo + 6 * 10 ** 6 + 10 ** 5).astype(np.int64)
    g = np.diff(p)
    for a in range(lo, lo + 6 * 10 ** 6, 20000):
        i, j = np.searchsorted(p, [a, a + 20000])
        k = i + int(np.argmax(g[i:j]))
        r = engine.sieve_range(a, a + 20000)
        assert (r["max_gap"], r["gap_start"]) == (int(g[k]), int(p[k])), a


def test_served(engine):
    with mp.Server(engine, streams=2) as srv:
        ids = [srv.submit_range(lo, hi) for _, lo, hi in TIES]
        for rid, (gap, lo, hi) in zip(ids, TIES):
            r = None
            while r is None:
                r = srv.poll(rid, 500)
            alone = engine.sieve_range(lo, hi, mode=mp.MODE_PLAIN)
            assert (r["max_gap"], r["gap_start"]) == (gap, alone["gap_start"])
