"""The base-2 strong test's windowed ladder against Python's integers where its cases meet: the
smallest moduli, odd parts of n - 1 too short for a window (n = d 2^s + 1), every length of the
first window, digits at both ends, and the limits of the two size classes (2^62, 2^64)."""
import ctypes as C
import random

import numpy as np
import pytest

import mathpub_b200 as mp

pytestmark = pytest.mark.gpu


def sprp2(n):
    if n < 3 or n % 2 == 0:
        return n == 2
    d, s = n - 1, 0
    while d % 2 == 0:
        d, s = d // 2, s + 1
    x = pow(2, d, n)
    return x in (1, n - 1) or any(pow(2, d << r, n) == n - 1 for r in range(1, s))


def gpu(ns):
    L = mp.lib()
    L.cu_init.argtypes = [C.c_char_p, C.c_size_t]
    L.cu_sprp_batch.argtypes = [C.c_void_p, C.c_size_t, C.c_void_p]
    name = C.create_string_buffer(128)
    assert L.cu_init(name, 128) == 0
    arr = np.zeros((len(ns), 2), dtype=np.uint64)
    arr[:, 0] = ns
    ok = np.zeros(len(ns), dtype=np.uint8)
    assert L.cu_sprp_batch(arr.ctypes.data, len(ns), ok.ctypes.data) == 0
    return [bool(x) for x in ok]


def short_odd_parts():
    return [d << s | 1 for d in list(range(1, 140, 2)) + [(1 << 20) + 1, (1 << 32) - 1] for s in range(1, 64)
            if d << s < 2 ** 64 - 1]


def windows():
    ns = list(range(3, 3000, 2))
    for b in range(6, 64):
        ns += [(1 << b) + o for o in range(-9, 11, 2)] + [((1 << b) // 31 | 1) + o for o in (-2, 0, 2)]
    return [n for n in ns if n > 2]


def class_limits():
    rng = random.Random(62)
    ns = []
    for c in (2 ** 61, 2 ** 62, 2 ** 63):
        ns += [c + o for o in range(-399, 400, 2)]
    ns += [2 ** 64 - o for o in range(1, 400, 2)]
    return ns + [rng.randrange(2 ** 61, 2 ** 64) | 1 for _ in range(3000)]


@pytest.mark.parametrize("cases", [short_odd_parts, windows, class_limits])
def test_verdicts(cases):
    ns = cases()
    assert gpu(ns) == [sprp2(n) for n in ns]
