"""Fermat quotients to host arrays around the size from which the array's pages are mapped ahead
(2^17 quotients): any alignment, nothing written beside the results, and nothing at all where a p is
out of range."""
import ctypes as C

import numpy as np
import pytest

import mathpub_b200 as mp

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng():
    with mp.Engine(0) as e:
        yield e


def call(eng, p, q, offset):
    return mp.lib().mp_fermat_q_base2(eng.handle, C.c_void_p(p.ctypes.data), len(p), C.c_void_p(q.ctypes.data + 8 * offset))


@pytest.mark.parametrize("count", [2 ** 17 - 1, 2 ** 17, 2 ** 17 + 1, 2 ** 18 + 513])
@pytest.mark.parametrize("offset", [0, 1, 511])
def test_offsets(eng, count, offset):
    p = eng.primes_range(10 ** 9, 10 ** 9 + 24 * count)[:count]
    assert len(p) == count
    q = np.full(count + 1024, 0xAAAA, dtype=np.uint64)
    assert call(eng, p, q, offset) == mp.MP_OK
    assert (q[:offset] == 0xAAAA).all() and (q[offset + count:] == 0xAAAA).all()
    for i in (0, 1, count // 2, count - 1):
        v = int(p[i])
        assert int(q[offset + i]) == (pow(2, v - 1, v * v) - 1) // v
    parts = np.concatenate([eng.fermat_quotient(p[k:k + 50000]) for k in range(0, count, 50000)])
    assert np.array_equal(q[offset:offset + count], parts)


def test_out_of_range_writes_nothing(eng):
    p = np.full(2 ** 17 + 5, 1000003, dtype=np.uint64)
    p[70000] = 2 ** 63 + 29
    q = np.full(len(p), 7, dtype=np.uint64)
    assert call(eng, p, q, 0) == mp.MP_ERANGE
    assert (q == 7).all()
