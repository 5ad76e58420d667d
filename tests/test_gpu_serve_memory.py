"""The memory that a served range is admitted with is what it takes: the buffers that a new handle allocates for
the range, less the room they keep to grow (1/16 of the planes and records, a third of the threads' state, 72 MB)."""
import ctypes as C

import pytest

import mathpub_b200 as mp

pytestmark = pytest.mark.gpu


def free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("lo,n", [(9 * 10 ** 17, 2 ** 32), (9 * 10 ** 17, 2 ** 20), (10 ** 15, 2 ** 34), (10 ** 12, 2 ** 30), (10 ** 9, 2 ** 16)])
def test_estimate(lo, n):
    f = mp.lib().mp_sieve_scratch
    f.argtypes, f.restype = [C.c_void_p, C.c_uint64, C.c_uint64], C.c_uint64
    with mp.Engine(0) as other:
        other.sieve_range(lo, lo + n)                      # kernels loaded
    with mp.Engine(0) as e:
        e.tune_set(tile_log2=18)
        e.sieve_range(lo + n - 1000, lo + n)               # tables, by another form's buffers
        e.tune_set(tile_log2=0)
        before = free()
        e.sieve_range(lo, lo + n)
        took, est = before - free(), f(e.handle, lo, lo + n)
    assert took - est / 3 - (80 << 20) <= est <= took + (64 << 20), (took, est)


def test_small_budget_serves_all():
    """Requests larger than the budget run one at a time."""
    lo, n = 9 * 10 ** 17, 2 ** 24
    with mp.Engine(0) as e:
        want = e.sieve_range(lo, lo + n)
        with mp.Server(e, streams=2, mem_budget=1 << 20) as srv:
            ids = [srv.submit_range(lo, lo + n) for _ in range(6)]
            for i in ids:
                r = None
                while r is None:
                    r = srv.poll(i, 500)
                assert r["status"] == mp.MP_OK and r["pi"] == want["pi"] and r["gap_start"] == want["gap_start"]
