"""The two forms of the segment hash (a warp per segment with the low byte's state found by prefix
XORs; a thread per segment) against FNV-1a in Python on the returned bitmap: segments below, at and
above a row of the parallel form, counts on both sides of the choice, and ranges whose last segment
ends inside a row, a word or a byte."""
import numpy as np
import pytest

from helpers import FNV_OFF, FNV_PRIME

pytestmark = pytest.mark.gpu


def fnv_segments(bits, seg_bits):
    """FNV-1a-64 of each run of seg_bits bits (the last one short), vectorised over the runs."""
    n = len(bits)
    ns = -(-n // seg_bits)
    h = np.full(ns, FNV_OFF, dtype=np.uint64)
    full = np.zeros(ns * seg_bits, dtype=np.uint8)
    full[:n] = bits
    by = np.packbits(full, bitorder="little").reshape(ns, -1)
    last = n - (ns - 1) * seg_bits                                # bits of the last segment
    for k in range(by.shape[1]):
        live = ns if 8 * k < last else ns - 1
        h[:live] = (h[:live] ^ by[:live, k]) * np.uint64(FNV_PRIME)
    return h


@pytest.mark.parametrize("lo,length,hash_log2", [
    (10 ** 9, 10 ** 6, 14),                 # 1024-byte segments: one row
    (10 ** 9 + 1, 10 ** 6 + 77, 13),        # 512-byte segments: the serial form
    (10 ** 12, 5 * 10 ** 6 + 3, 19),        # 32 KiB, the last segment short by bits
    (10 ** 12, 2 ** 20 + 2 * 8 * 1000, 20),  # a last segment of 1000 bytes
    (7 * 10 ** 13, 2 ** 20 + 2, 20),        # a last segment of one bit
    (10 ** 10, 11000 * 2 ** 14, 14),        # the parallel form's largest count
    (10 ** 10, 11001 * 2 ** 14 - 6, 14),    # one more: the serial form, last segment short
    (123456789, 3 * 10 ** 5, 8), (10 ** 9, 4096, 4)])
def test_hash_forms(engine, lo, length, hash_log2):
    r = engine.sieve_range(lo, lo + length, hash_log2=hash_log2, bitmap=True)
    nbits = (lo + length - (lo & ~1)) >> 1
    bits = np.unpackbits(r["bitmap"].view(np.uint8), bitorder="little")[:nbits]
    assert np.array_equal(r["hashes"], fnv_segments(bits, 1 << (hash_log2 - 1)))
