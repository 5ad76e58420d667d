"""Prime lists where a warp's window of 30720 integers holds more primes than its part of shared memory: a build
of the library with a part of 1000 primes (windows near 1e9 hold 1480, near 1e18 740) gives the oracle's lists,
whole ones and ones that end at a given capacity."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import ctypes as C, sys
sys.path.insert(0, sys.argv[2])
import numpy as np
import mathpub_b200 as mp, oracle
mp.LIB_PATH = sys.argv[1]
oracle.o()
with mp.Engine(0) as e:
    for lo, n in ((0, 100000), (10 ** 9 + 7, 3 * 10 ** 6), (10 ** 13, 2 ** 22), (10 ** 18, 2 ** 21)):
        want = oracle.primes_range(lo, lo + n)
        assert np.array_equal(e.primes_range(lo, lo + n), want), lo
        cap = len(want) * 2 // 3
        out, cnt = np.full(cap + 8, 7, dtype=np.uint64), C.c_size_t()
        assert mp.lib().mp_primes_range(e.handle, lo, lo + n, C.c_void_p(out.ctypes.data), cap, C.byref(cnt)) == 0
        assert cnt.value == len(want) and np.array_equal(out[:cap], want[:cap]) and (out[cap:] == 7).all()
print("same")
"""


def test_rows_past_their_part(orc, tmp_path):
    from mathpub_b200 import build
    lib = str(tmp_path / "libsmallrows.so")
    src = [os.path.join(build.CSRC, s) for s in build.SOURCES]
    r = subprocess.run([build.NVCC, *build.FLAGS, "-DEMIT_ROW=1000u", "-shared", "-o", lib, *src], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([sys.executable, "-c", CHILD, lib, ROOT], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "same" in r.stdout, r.stderr
