"""floor(w 2^64 / q) by digits of 32 bits, on the host: the code the kernels run.

Moduli from 3 to 62 bits (powers of two and their neighbours, upper halves of all
ones and of one bit, NTT primes), operands at the edges of [0, q) and random ones,
against whole numbers.
"""
import ctypes as C
import os
import random
import subprocess

import pytest

from anns_fhe_b200.build import CSRC
from anns_fhe_b200.driver import find_ntt_primes


@pytest.fixture(scope="module")
def companion(tmp_path_factory):
    d = tmp_path_factory.mktemp("companion")
    src, so = os.path.join(d, "c.cpp"), os.path.join(d, "c.so")
    with open(src, "w") as f:
        f.write('#include "modarith.cuh"\n'
                'extern "C" uint64_t companion(uint64_t w, uint64_t q) { return afhe::shoup_companion(w, q); }\n')
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, "-x", "c++", src, "-o", so], check=True)
    f = C.CDLL(so).companion
    f.restype, f.argtypes = C.c_uint64, [C.c_uint64, C.c_uint64]
    return f


def test_companion(companion):
    rng = random.Random(5)
    qs = [3, 5, 7]
    for b in range(2, 62):
        qs += [(1 << b) - 1, 1 << b, (1 << b) + 1, (1 << b) | rng.getrandbits(b), (1 << b) | rng.getrandbits(max(1, b // 2))]
        qs += [((1 << b + 1) - 1) ^ rng.getrandbits(max(1, b - 32))]
    for b in (30, 36, 49, 50, 60, 61):
        qs += find_ntt_primes(13, b, 2, [])
    for q in qs:
        edges = [0, 1, 2, q // 2, q // 2 + 1, q - 2, q - 1, (1 << 32) - 1, 1 << 32, (1 << 32) + 1]
        for w in [x for x in edges if 0 <= x < q] + [rng.randrange(q) for _ in range(60)]:
            assert companion(w, q) == (w << 64) // q, (w, q)
