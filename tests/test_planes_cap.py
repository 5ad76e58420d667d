"""The capacity of a tile's bucket (mathpub_b200/csrc/mp_planes_cap.h) against the exact numbers of records in the
148 blocks of a first wave, for ranges from 0 and from near 0, where a few cofactors u of the multiples q u
decide how many primes hit a block.  CPU only; the range [0, 3e13) on the GPU."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HEADER = os.path.join(ROOT, "mathpub_b200", "csrc", "mp_planes_cap.h")

PT = 1769472                               # the largest tile, which long ranges take
NB = 148                                   # blocks of a wave
RES = (1, 7, 11, 13, 17, 19, 23, 29)


@pytest.fixture(scope="module")
def cap(tmp_path_factory):
    d = tmp_path_factory.mktemp("cap")
    src, so = str(d / "cap.c"), str(d / "cap.so")
    with open(src, "w") as f:
        f.write(f'#include "{HEADER}"\n'
                "uint32_t cap(uint32_t pt, double s, uint64_t i0, uint32_t q) { return plane_bucket_cap(pt, s, i0, q); }\n")
    subprocess.run([os.environ.get("CC", "gcc"), "-O1", "-shared", "-fPIC", "-o", so, src, "-lm"], check=True)
    f = C.CDLL(so).cap
    f.argtypes = [C.c_uint32, C.c_double, C.c_uint64, C.c_uint32]
    f.restype = C.c_uint32
    return f


@pytest.fixture(scope="module")
def primes():
    n = 10 ** 8
    s = np.ones(n // 2, dtype=bool)
    for i in range(3, int(n ** 0.5) + 1, 2):
        if s[i // 2]:
            s[i * i // 2:: i] = False
    s[0] = False
    return 2 * np.flatnonzero(s).astype(np.int64) + 1


def most_records(q, i0):
    """The largest number of multiples q k of the primes q, other than q itself, in a block of a plane."""
    most = 0
    qa, c = q // 30, q % 30
    inv = c * c % 30 * c % 30
    for r in RES:
        u = r * inv % 30
        j = qa * u + (c * u - r) // 30 - i0 % q
        j[j < 0] += q[j < 0]
        own = (u == 1) & (i0 + j == qa)
        j[own] += q[own]
        n, qq = np.zeros(NB, dtype=np.int64), q
        while len(j):
            keep = j < NB * PT
            j, qq = j[keep], qq[keep]
            n += np.bincount(j // PT, minlength=NB)
            j = j + qq
        most = max(most, int(n.max()))
    return most


@pytest.mark.parametrize("lo", [0, 10 ** 7, 3 * 10 ** 7, 10 ** 9])
@pytest.mark.parametrize("hi", [10 ** 13, 3 * 10 ** 13, 10 ** 14, 10 ** 15, 10 ** 16])
def test_first_wave_fits(cap, primes, lo, hi):
    q = primes[(primes > PT * 3 // 2) & (primes <= hi ** 0.5)]
    c = cap(PT, float((1.0 / q).sum()), lo // 30, int(q[-1]))
    assert most_records(q, lo // 30) <= c


def test_far_from_zero_nothing_is_added(cap):
    """[1e15, +2^34): the 2%, the square root and 256, to a record."""
    e = PT * 0.15488
    assert abs(cap(PT, 0.15488, 10 ** 15 // 30, 31622777) - (1.02 * e + 10 * (e + 1) ** 0.5 + 256)) < 4


@pytest.mark.gpu
def test_range_from_zero(engine):
    hi, cut = 3 * 10 ** 13, 10 ** 13
    whole = engine.sieve_range(0, hi)
    a, b = engine.sieve_range(0, cut), engine.sieve_range(cut, hi)
    for k in ("pi", "twins", "tuple6"):
        assert whole[k] == a[k] + b[k], k
    assert whole["max_gap"] == max(a["max_gap"], b["max_gap"])
