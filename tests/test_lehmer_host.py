"""The Lehmer rounds of a gcd (mersenne_trinomial_b200/csrc/lehmer.cuh) in a
block on the host, its warps run in every order that its barriers leave open
for one of them: warp 0, which decides each round, as early or as late as it
can, and each of the others last.  Results against Euclid on whole numbers
and, for the half-gcd's rounds, the matrix against the vector it gives."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "mersenne_trinomial_b200", "csrc")
TESTS = os.path.join(ROOT, "tests")
WARPS = 16


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("lehmer")
    shutil.copy(os.path.join(CSRC, "lehmer.cuh"), d)
    shutil.copy(os.path.join(TESTS, "cta_host.h"), os.path.join(d, "gf2e_internal.cuh"))
    shutil.copy(os.path.join(TESTS, "lehmer_driver.cpp"), d)
    so = os.path.join(d, "lehmer.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-Wno-unknown-pragmas",
                    "-I" + os.path.join(ROOT, "include"), "-o", so,
                    os.path.join(d, "lehmer_driver.cpp")], check=True, timeout=300)
    return C.CDLL(so)


def _order(first, last):
    rest = [w for w in range(WARPS) if w not in (first, last)]
    return [first] + rest + ([last] if last != first else [])


def _words(v, n):
    return [(v >> (64 * i)) & (2**64 - 1) for i in range(n)]


def _value(words):
    return sum(int(w) << (64 * i) for i, w in enumerate(words))


def _gcd(a, b):
    while b:
        while a.bit_length() >= b.bit_length() and a:
            a ^= b << (a.bit_length() - b.bit_length())
        a, b = b, a
    return a


def _mul(a, b):
    r = 0
    while b:
        low = b & -b
        r ^= a << (low.bit_length() - 1)
        b ^= low
    return r


def _poly(bits, seed):
    v = int.from_bytes(np.random.default_rng(seed).bytes(bits // 8 + 1), "little")
    return v & ((1 << bits) - 1) | 1 << (bits - 1)


def _run(lib, a, b, order, m=0, mw=0):
    W = max(a.bit_length(), b.bit_length()) // 64 + 2
    V = np.array(_words(a, W) + _words(b, W) + [0] * (2 * W), dtype=np.uint64)
    R = np.zeros(8 * mw, dtype=np.uint64)
    if mw:
        R[0] = R[3 * mw] = 1
    out = [C.c_int() for _ in range(3)]
    rounds = C.c_longlong()
    st = lib.lehmer_host(V.ctypes.data_as(C.c_void_p), C.c_uint64(W),
                         R.ctypes.data_as(C.c_void_p) if mw else None, C.c_uint64(mw),
                         C.c_longlong(a.bit_length() - 1), C.c_longlong(b.bit_length() - 1),
                         C.c_longlong(m), (C.c_int * WARPS)(*order), *[C.byref(o) for o in out],
                         C.byref(rounds))
    va, ra, parity = (o.value for o in out)
    return st, _value(V[va * W:(va + 1) * W]), R, ra, parity, rounds.value


PAIRS = [(700, 650, 65), (1500, 1400, 130), (900, 200, 65), (400, 33, 1), (64, 64, 1), (130, 3, 2)]


@pytest.mark.parametrize("first,last", [(0, w) for w in range(1, WARPS)] + [(5, 0), (1, 15)])
def test_gcd_in_any_warp_order(lib, first, last):
    for i, (ab, bb, common) in enumerate(PAIRS):
        c = _poly(common, 40 + i)
        a, b = _mul(_poly(ab - common + 1, i), c), _mul(_poly(bb - common + 1, 20 + i), c)
        st, g, *_ = _run(lib, a, b, _order(first, last))
        assert st == 0, (ab, bb, st)
        assert g == _gcd(a, b), (ab, bb)


@pytest.mark.parametrize("first,last", [(0, 1), (0, 7), (0, 15), (3, 0)])
def test_matrix_in_any_warp_order(lib, first, last):
    for i, (ab, bb) in enumerate([(1400, 1399), (900, 860), (2000, 1100)]):
        a, b = _poly(ab, 60 + i), _poly(bb, 70 + i)
        m, mw = ab // 2, ab // 128 + 4
        st, v, R, ra, parity, _ = _run(lib, a, b, _order(first, last), m, mw)
        assert st == 0 and v.bit_length() - 1 >= m
        row = parity * 4 + 2 * ra
        e = [_value(R[(row + k) * mw:(row + k + 1) * mw]) for k in range(2)]
        assert _mul(e[0], a) ^ _mul(e[1], b) == v, (ab, bb)


# a gcd with 1, or that comes down to 1, ends there: no round for each
# coefficient of the other operand
@pytest.mark.parametrize("bits", [1, 64, 65, 3000])
def test_unit_operand_takes_no_rounds(lib, bits):
    a = _poly(bits, bits)
    for x, y in ((a, 1), (1, a)):
        st, g, *_, rounds = _run(lib, x, y, _order(0, 15))
        assert (st, g) == (0, 1)
        assert rounds == 0
    a = _mul(_poly(2000, 9), 0b10) ^ 1              # a = 1 mod x
    st, g, *_, rounds = _run(lib, a, 0b10, _order(0, 15))
    assert (st, g) == (0, 1)
    assert rounds <= 2 * 2000
