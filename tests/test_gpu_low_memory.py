"""Calls on a device with little free memory: one that cannot have its tables fails with MP_ENOMEM and leaves the
handle as it was, so that the same call succeeds once there is memory."""
import numpy as np
import pytest

import mathpub_b200 as mp

pytestmark = pytest.mark.gpu

SEXT = (0, 4, 6, 10, 12, 16)


class Ballast:
    """Holds the device's free memory but for `leave` bytes."""

    def __init__(self, leave):
        self.leave, self.held = leave, []

    def __enter__(self):
        import torch
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        size = 1 << 36
        while size >= 1 << 21:
            free = torch.cuda.mem_get_info()[0] - self.leave
            if free >= size + (1 << 22):
                try:
                    self.held.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
                    continue
                except torch.OutOfMemoryError:
                    pass
            size >>= 1
        return self

    def __exit__(self, *a):
        import torch
        self.held.clear()
        torch.cuda.empty_cache()


def enomem(call):
    with pytest.raises(mp.MathpubError) as x:
        call()
    assert x.value.code == mp.MP_ENOMEM


def test_constellation_tables():
    lo, n = 10 ** 15, 10 ** 12
    with mp.Engine(0) as other:
        want = other.tuple_count(lo, lo + n, SEXT), other.chain_sieve(lo, lo + n, 10)
    with mp.Engine(0) as e:
        e.sieve_range(10 ** 9, 10 ** 9 + 1000)
        with Ballast(4 << 20):
            enomem(lambda: e.tuple_count(lo, lo + n, SEXT))
            enomem(lambda: e.tuple_count(lo, lo + n, SEXT))
        assert e.tuple_count(lo, lo + n, SEXT) == want[0]
        with Ballast(4 << 20):                               # a plan on the handle, no room for another beside it
            try:
                h, l = e.chain_sieve(lo, lo + n, 10)
                assert np.array_equal(h, want[1][0]) and np.array_equal(l, want[1][1])
            except mp.MathpubError as x:
                assert x.code == mp.MP_ENOMEM
        h, l = e.chain_sieve(lo, lo + n, 10)
        assert np.array_equal(h, want[1][0]) and np.array_equal(l, want[1][1])
        assert e.tuple_count(lo, lo + n, SEXT) == want[0]


def test_two_plans_share_the_work_lists():
    """Two patterns used in turn on one handle hold the work lists once (about 0.5 GB here), not once each."""
    import torch
    lo, n = 10 ** 15, 2 * 10 ** 11

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    with mp.Engine(0) as other:
        want = other.tuple_count(lo, lo + n, (0, 2, 6, 8)), other.tuple_count(lo, lo + n, (0, 4, 6, 10))
    with mp.Engine(0) as e:
        before = free()
        assert e.tuple_count(lo, lo + n, (0, 2, 6, 8)) == want[0]
        one = free()
        assert e.tuple_count(lo, lo + n, (0, 4, 6, 10)) == want[1]
        two = free()
        assert before - one > 200 << 20 and one - two < 100 << 20
        for _ in range(2):
            assert e.tuple_count(lo, lo + n, (0, 2, 6, 8)) == want[0]
            assert e.tuple_count(lo, lo + n, (0, 4, 6, 10)) == want[1]
        assert two - free() < 32 << 20


def stats(r):
    return {k: r[k] for k in ("pi", "twins", "max_gap", "gap_start", "tuple6", "tuple6_cks", "first_prime", "last_prime")}


def range_with(lo, n, leave):
    """A range on a new handle, with `leave` bytes of device memory beside its tables."""
    with mp.Engine(0) as other:
        want = other.sieve_range(lo, lo + n)
    with mp.Engine(0) as e:
        e.sieve_range(lo + n - 2 ** 16, lo + n)
        with Ballast(leave):
            got = [e.sieve_range(lo, lo + n) for _ in range(4)]         # the later ones captured and replayed
        assert all(stats(r) == stats(want) for r in got)
        assert stats(e.sieve_range(lo, lo + n)) == stats(want)


def test_range_without_room_to_spare():
    """A wave's buffers take about 80 MB here, and half as much again with what they grow by beyond the need."""
    range_with(10 ** 12, 2 ** 30, 60 << 20)


@pytest.mark.parametrize("leave_mb", [1000, 400])
def test_range_in_shorter_waves(leave_mb):
    """One wave's buffers take 1.9 GB here."""
    range_with(9 * 10 ** 17, 2 ** 32, leave_mb << 20)


def test_prime_list_of_its_exact_size():
    """The 1.63 GB of the primes below 2^32 fit, the 1.95 GB of the bound on their number do not."""
    hi = 2 ** 32
    with mp.Engine(0) as other:
        want = other.wieferich_range(0, hi)
    with mp.Engine(0) as e:
        e.sieve_range(0, hi)                                          # the sieve's own buffers
        with Ballast(1780 << 20):
            got = e.wieferich_range(0, hi)
    assert got == want
