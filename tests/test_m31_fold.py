"""The M31 folds of csrc/m31.cuh, whose functions are the same on the host and the device, compiled
here for the host and compared with integers (exact arithmetic: tolerance zero)."""
import ctypes
import itertools
import os
import random
import subprocess

import pytest

from gkr_gb300 import build as libbuild
from gkr_gb300 import circuit as gc

P = gc.P

SOURCE = """
#include "m31.cuh"
extern "C" uint32_t lerp(uint32_t a, uint32_t b, uint32_t r) { return m31::lerp(a, b, m31::lerp_at(r)); }
extern "C" uint32_t lerp2(const uint32_t* x, uint32_t r0, uint32_t r1) {
    return m31::lerp2(x[0], x[1], x[2], x[3], m31::lerp2_at(r0, r1));
}
extern "C" uint32_t weighted(const uint32_t* x, const uint32_t* c) {
    const m31::Lerp2 w = {{c[0], c[1], c[2], c[3]}};
    return m31::lerp2(x[0], x[1], x[2], x[3], w);
}
"""


@pytest.fixture(scope="module")
def m31(tmp_path_factory):
    d = tmp_path_factory.mktemp("m31")
    (d / "m31_host.cpp").write_text(SOURCE)
    subprocess.check_call([os.environ.get("CXX", "g++"), "-std=c++17", "-O2", "-Wall", "-fPIC", "-shared", "-I",
                           libbuild.CSRC, str(d / "m31_host.cpp"), "-o", str(d / "m31_host.so")])
    return ctypes.CDLL(str(d / "m31_host.so"))


def call(f, *args):
    f.restype = ctypes.c_uint32
    return f(*[(ctypes.c_uint32 * len(a))(*a) if isinstance(a, (list, tuple)) else ctypes.c_uint32(a) for a in args])


def fold(a, b, r):
    return (a + (b - a) * r) % P


def fold2(x, r0, r1):
    return fold(fold(x[0], x[1], r0), fold(x[2], x[3], r0), r1)


@pytest.mark.parametrize("x,r0,r1", [
    # totals whose parts of 31, 31 and 2 bits add to 2p or more
    ((367724859, 1697068605, 2122615719, 1832151202), 1353201603, 398097677),
    ((944683800, 1267107643, 1303277034, 960102954), 1882670236, 839795476),
])
def test_two_folds_of_the_largest_parts(m31, x, r0, r1):
    assert call(m31.lerp2, x, r0, r1) == fold2(x, r0, r1)


def factors(total):
    """Canonical x and c whose four products add to `total`: the first three weights are P - 1, the
    last a prime by which what is left divides for one of as many values of x0 + x1 + x2."""
    for c3 in (1, 65521, 2147483629):
        first = max(0, -(-(total - c3 * (P - 1)) // (P - 1)))
        q = first + (total * pow(P - 1, -1, c3) - first) % c3 if c3 > 1 else first
        left = total - q * (P - 1)
        if q <= 3 * (P - 1) and left >= 0 and left % c3 == 0 and left // c3 < P:
            x0, x1 = min(q, P - 1), min(max(q - (P - 1), 0), P - 1)
            return [x0, x1, q - x0 - x1, left // c3], [P - 1, P - 1, P - 1, c3]
    raise AssertionError("no factors")


@pytest.mark.parametrize("hi", [0, 1, 0x3FFFFFFF, 0x40000000, 0x7FFFFFFE, 0x7FFFFFFF, 0x80000000, 0xBFFFFFFE, 0xBFFFFFFF,
                                0xC0000000])
def test_sums_of_four_products_at_the_ends_of_their_words(m31, hi):
    for lo in (0, 1, 0x7FFFFFFD, 0x7FFFFFFE, 0x7FFFFFFF, 0x80000000, 0xFFFFFFFC, 0xFFFFFFFD, 0xFFFFFFFE, 0xFFFFFFFF):
        total = hi << 32 | lo
        x, c = factors(total)
        assert sum(a * b for a, b in zip(x, c)) == total and max(x + c) < P
        assert call(m31.weighted, x, c) == total % P, hex(total)
    assert call(m31.weighted, [P - 1] * 4, [P - 1] * 4) == 4  # the largest sum


def test_folds_of_edge_and_random_values(m31):
    edge = [0, 1, 2, P // 2, P // 2 + 1, P - 2, P - 1]
    for a, b, r in itertools.product(edge, repeat=3):
        assert call(m31.lerp, a, b, r) == fold(a, b, r)
    rng = random.Random(71)
    for _ in range(20000):
        v = [rng.choice(edge) if rng.random() < 0.5 else rng.randrange(P) for _ in range(6)]
        assert call(m31.lerp2, v[:4], v[4], v[5]) == fold2(v[:4], v[4], v[5])
