"""Segment hashes of a bitmap that the caller placed 4, 8 or 12 bytes past a 16-byte boundary equal those of an
aligned one, in both forms and with a last segment of any length."""
import ctypes as C

import numpy as np
import pytest

import mathpub_b200 as mp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lo,length,hash_log2", [
    (10 ** 12, 11500 * 2 ** 14 + 77, 14),   # many segments: a thread each
    (10 ** 12, 11500 * 2 ** 13, 13), (10 ** 9, 3 * 10 ** 6 + 3, 8), (10 ** 9, 5000, 4),
    (10 ** 12, 40 * 2 ** 19 + 2, 19)])      # few: a warp each
def test_offsets(engine, lo, length, hash_log2):
    import torch
    L = mp.lib()
    hi = lo + length
    want = engine.sieve_range(lo, hi, hash_log2=hash_log2, bitmap=True)
    nw, nh = L.mp_sieve_nwords(lo, hi), L.mp_sieve_nhashes(lo, hi, hash_log2)
    o = mp.SieveOpts(mp.MODE_BATCHED, 0, 0, hash_log2, 0)
    st = torch.cuda.current_stream().cuda_stream
    for off in (0, 4, 8, 12):
        bm = torch.zeros(nw * 8 + 64, dtype=torch.uint8, device="cuda")
        hs = torch.zeros(nh, dtype=torch.int64, device="cuda")
        out = torch.zeros(64, dtype=torch.int64, device="cuda")
        assert bm.data_ptr() % 16 == 0
        rc = L.mp_sieve_range_dev(engine.handle, C.c_uint64(lo), C.c_uint64(hi), C.byref(o), C.c_void_p(out.data_ptr()), None,
                                  C.c_void_p(hs.data_ptr()), C.c_void_p(bm.data_ptr() + off), C.c_void_p(st))
        torch.cuda.synchronize()
        assert rc == mp.MP_OK
        assert np.array_equal(hs.cpu().numpy().view(np.uint64), want["hashes"]), off
        assert np.array_equal(bm[off:off + nw * 8].cpu().numpy().view(np.uint64), want["bitmap"]), off
