"""The multiply instructions behind bench.py's multiply-pipe rooflines: the squarings, shifts and their counts of
the base-2 and Fermat ladders against loops written as the kernels' are, and the instructions of each part against
the multiplies in its PTX block (CPU)."""
import os
import re
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)
import bench  # noqa: E402


def ladder_base2(n):
    d = n - 1
    while d % 2 == 0:
        d //= 2
    w = (n.bit_length() - 4) // 5 if n.bit_length() > 8 else 0
    while d >> (5 * w) == 0:
        w -= 1
    c = d >> (5 * w)
    squarings = shifts = 0
    c -= min(c, 63)
    while c:
        shifts += 1
        c -= min(c, 32)
    while w > 0:
        w -= 1
        squarings += 5
        shifts += 1
    return squarings * bench.IMAD_PER_SQUARING_BASE2[n >> 63] + shifts * bench.IMAD_PER_SHIFT_BASE2


def test_base2_ladder():
    rng = np.random.default_rng(3)
    n = np.concatenate([np.arange(3, 3000, 2, dtype=np.uint64)] +
                       [rng.integers(1 << (b - 1), 1 << b, 50, dtype=np.uint64) | np.uint64(1) for b in range(8, 65)] +
                       [np.array([(1 << b) + 1 for b in range(2, 64)] + [2 ** 64 - 1, 2 ** 63 + 1], dtype=np.uint64)])
    assert bench.base2_multiplies(n).tolist() == [ladder_base2(int(x)) for x in n]


def test_fermat_ladder():
    for bits in range(2, 48):
        t = bits - 6 if bits > 6 else 0
        w, rem = t // 5, t % 5
        want = t * bench.IMAD_PER_SQUARING_FERMAT_K3 + (w + (rem > 0)) * bench.IMAD_PER_SHIFT_FERMAT_K3
        assert bench.fermat_multiplies_k3(bits) == want + bench.IMAD_LEAVE_FERMAT_K3


def multiplies(name, opening, which=0):
    text = open(os.path.join(ROOT, "mathpub_b200", "csrc", name)).read()
    body = text[text.index(opening):]
    block = re.findall(r"asm\((.*?)\n +: \"", body, re.S)[which]
    return len(re.findall(r"\"(?:mul|mad|madc)\.", block))


@pytest.mark.parametrize("name,opening,which,want", [
    ("mp_mont64.cuh", "__device__ __forceinline__ void sp_sqr(", 0, bench.IMAD_PER_SQUARING_BASE2[0]),
    ("mp_mont64.cuh", "__device__ __forceinline__ void sp_sqr(", 1, bench.IMAD_PER_SQUARING_BASE2[1]),
    ("mp_mont64.cuh", "__device__ __forceinline__ void sp_shift(", 0, bench.IMAD_PER_SHIFT_BASE2),
    ("mp_fermat.cu", "__device__ __forceinline__ void msqr<3>(", 0, bench.IMAD_PER_SQUARING_FERMAT_K3),
    ("mp_fermat.cu", "__device__ __forceinline__ void mshift<3>(", 0, bench.IMAD_PER_SHIFT_FERMAT_K3)])
def test_instructions_of_a_part(name, opening, which, want):
    assert multiplies(name, opening, which) == want
