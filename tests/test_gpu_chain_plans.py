"""The constellation sieve's plans by range length (two wheels, two pattern depths) and the last
segment's early end: chains and sextuplets of a long range equal those of its parts, which run under
another plan, and the plan kept for the other length serves again."""
import pytest

pytestmark = pytest.mark.gpu

SEXT = (0, 4, 6, 10, 12, 16)
M = 2 ** 64


@pytest.mark.parametrize("lo,length,parts", [(10 ** 13, 2 ** 40 + 12345, 5), (10 ** 15 + 7, 6 * 10 ** 12, 13)])
def test_sextuplets_add_up(engine, lo, length, parts):
    n, c = engine.tuple_count(lo, lo + length, SEXT)
    cut = [lo + length * i // parts for i in range(parts + 1)]
    got = [engine.tuple_count(a, b, SEXT) for a, b in zip(cut, cut[1:])]
    assert (n, c) == (sum(x for x, _ in got), sum(x for _, x in got) % M)


@pytest.mark.parametrize("k,dec,lo,length", [(9, False, 10 ** 14, 6 << 44), (10, True, 3 * 10 ** 15, (6 << 44) + 99991),
                                             (11, False, 10 ** 17, 2 * 10 ** 14)])
def test_chains_of_the_parts(engine, k, dec, lo, length):
    h, l = engine.chain_sieve(lo, lo + length, k, dec=dec)
    cut = [lo + length * i // 4 for i in range(5)]
    want = []
    for a, b in zip(cut, cut[1:]):
        ph, pl = engine.chain_sieve(a, b, k, dec=dec)
        want += list(zip(ph.tolist(), pl.tolist()))
    assert sorted(zip(h.tolist(), l.tolist())) == sorted(want) and len(want) > 0
    h2, l2 = engine.chain_sieve(lo, lo + length, k, dec=dec)
    assert h2.tolist() == h.tolist() and l2.tolist() == l.tolist()
