"""mp_fermat_q_base2_dev with d_q = d_p: the quotients of composites, which are taken in a second look at the
entry, equal those written to another array, on both limb counts and one or two numbers a thread."""
import ctypes as C

import numpy as np
import pytest

import mathpub_b200 as mp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ilp2", [0, 1])
@pytest.mark.parametrize("lo,count", [(1, 1001), (10 ** 6 + 1, 2048), (2 ** 47 - 1001, 3001), (2 ** 62 + 1, 777)])
def test_in_place(lo, count, ilp2):
    import torch
    p = np.arange(lo, lo + count, dtype=np.uint64)               # even and odd, primes and composites
    p[::7] |= np.uint64(1)
    with mp.Engine(0) as e:
        e.tune_set(fermat_ilp2=ilp2)
        want = e.fermat_quotient(p)
        d = torch.from_numpy(p.view(np.int64).copy()).cuda()
        st = torch.cuda.current_stream().cuda_stream
        rc = mp.lib().mp_fermat_q_base2_dev(e.handle, C.c_void_p(d.data_ptr()), C.c_size_t(count), C.c_void_p(d.data_ptr()),
                                            C.c_void_p(st))
        torch.cuda.synchronize()
        assert rc == mp.MP_OK
        got = d.cpu().numpy().view(np.uint64)
    assert np.array_equal(got, want)
    odd = [int(x) for x in p if x % 2 and x >= 3][:200]
    for x in odd:
        q = (pow(2, x - 1, x * x) - 1) * pow(x, -1, 2 ** 64) % 2 ** 64
        assert int(got[int(np.flatnonzero(p == x)[0])]) == (q if q < x else 2 ** 64 - 1)
