"""The kernels' straight-line FP64 quotient, reciprocal and square root
(common.cuh) against IEEE's, bit for bit, over the ranges that their comment
states: random operands, all-ones and nearly all-ones significands, divisors
around powers of two, zero numerators, the ends of the ranges, and quotients as
close to the midpoint of two numbers as a pair of doubles allows -- those also
for divisors whose reciprocal is itself next to a midpoint, where the
reciprocal that the quotient starts from may be the wrong neighbour.

The bound that goes with the method: with b in [1, 2) the corrected quotient is
off by at most b 2^-108 (1 + 2^-7)^2 before its rounding, and a quotient of two
doubles that is no midpoint lies 2^-106 / b or more from one.  So the bits are
IEEE's for every b up to 2 (1 - 2^-7), and above it for all quotients but those
at the least distance, which may be the other neighbour."""
import ctypes
import os
import random
import subprocess
from fractions import Fraction

import numpy as np
import pytest

from eu3d_b200 import build

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))
ONE = 1 << 52


def _random(rng, n, e0, e1):
    m = rng.integers(ONE, 2 * ONE, n).astype(np.float64)
    return np.ldexp(m, rng.integers(e0, e1 + 1, n) - 52) * np.where(rng.random(n) < 0.5, -1.0, 1.0)


def operands_random():
    rng = np.random.default_rng(1)
    return _random(rng, 1 << 21, -300, 300), _random(rng, 1 << 21, -300, 300)


def operands_special():
    """Significands next to all ones and next to one, each over each, at several scales."""
    m = np.concatenate([2 * ONE - 1 - np.arange(400), ONE + np.arange(400), (3 * ONE) // 2 + np.arange(-50, 50)])
    a, b = np.meshgrid(m.astype(np.float64), m.astype(np.float64))
    a, b = np.ldexp(a.ravel(), -52), np.ldexp(b.ravel(), -52)
    return (np.concatenate([np.ldexp(a, s) for s in (0, 1, 77)]), np.concatenate([np.ldexp(b, s) for s in (0, -3, 300)]))


def operands_ends():
    """Both ends of the stated ranges (the quotient stays normal), and zero."""
    rng = np.random.default_rng(2)
    n = 1 << 16
    a = [_random(rng, n, -968, -960), _random(rng, n, -968, -960), _random(rng, n, 1010, 1023), _random(rng, n, -10, 10),
         _random(rng, n, -10, 10), np.zeros(n)]
    b = [_random(rng, n, -1000, -990), _random(rng, n, 0, 50), _random(rng, n, 20, 999), _random(rng, n, -1000, -990),
         _random(rng, n, 990, 999), _random(rng, n, -1000, 999)]
    return np.concatenate(a), np.concatenate(b)


def _near_midpoint(b):
    """Numerators a (integers of 53 bits) whose quotient by the odd integer b lies
    within |c| / (2^j b) of a midpoint m / 2^j, c = +-1, +-2, +-3: m is an odd
    integer of 54 bits, j = 54 for quotients below one and 53 above."""
    out = []
    for j, top in ((54, 0), (53, 1 << 53)):
        inv = pow(b, -1, 1 << j)
        for c in (1, -1, 2, -2, 3, -3):
            m = (-c * inv) % (1 << j) + top
            a = (m * b + c) >> j
            if m & 1 and m >> 53 == 1 and a >> 52 == 1:
                assert (a << j) - m * b == c
                out.append(a)
    return out


def operands_midpoint():
    rng = random.Random(3)
    a, b = [], []

    def add(d):
        for x in _near_midpoint(d):
            a.append(x)
            b.append(d)

    for _ in range(20000):
        add(rng.randrange(ONE, 2 * ONE) | 1)
    # 1 / d within 2^-7 of half an ulp of a midpoint, over all divisors and next to two
    for lo, n in ((ONE, 300000), (2 * ONE - (ONE >> 6), 300000), (2 * ONE - (1 << 20), 100000)):
        for _ in range(n):
            d = rng.randrange(lo, 2 * ONE) | 1
            if d == 2 * ONE - 1:
                continue
            frac = ((1 << 112) // d) & 0x7F  # 1/d scaled: 2^112/d has 60 bits, 53 of them the significand
            if frac in (0x3F, 0x40):
                add(d)
    for d in range(2 * ONE - 401, 2 * ONE, 2):
        add(d)
    return np.array(a, dtype=np.float64), np.array(b, dtype=np.float64)


CASES = {"random": operands_random, "special": operands_special, "ends": operands_ends, "midpoint": operands_midpoint}


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("quotients") / "libquotients.so")
    subprocess.run([os.environ.get("NVCC", "nvcc")] + build.NVCC_FLAGS + [os.path.join(HERE, "quotients.cu"), "-o", so],
                   check=True)
    return ctypes.CDLL(so)


@pytest.mark.parametrize("name", CASES)
def test_bits_of_ieee(lib, name):
    a, b = CASES[name]()
    a, b = np.ascontiguousarray(a), np.ascontiguousarray(b)
    assert len(a) == len(b) and np.all(np.abs(b) >= 2.0**-1000) and np.all(np.abs(b) <= 2.0**1000)
    with np.errstate(all="ignore"):
        want = (a / b, 1.0 / np.abs(b), np.sqrt(np.abs(a)))
    normal = (np.abs(want[0]) >= 2.0**-1022) & np.isfinite(want[0]) | (a == 0)
    assert normal.all()
    got = [np.empty_like(a) for _ in range(3)]
    ptr = [x.ctypes.data_as(ctypes.c_void_p) for x in (a, b, *got)]
    assert lib.quotients(ptr[0], ptr[1], ctypes.c_longlong(len(a)), *ptr[2:]) == 0
    for what, g, w, keep in zip(("quotient", "reciprocal", "root"), got, want,
                                (slice(None), slice(None), (np.abs(a) >= 2.0**-960) | (a == 0))):
        bad = [(x, y, u, v) for x, y, u, v in zip(*(z[keep][g[keep] != w[keep]] for z in (a, b, g, w)))]
        if what == "quotient":
            bad = [t for t in bad if not _other_neighbour(*t)]
        assert not bad, (what, len(bad), len(a), [[x.hex() for x in t] for t in bad[:3]])


def _other_neighbour(a, b, got, want):
    """Whether a / b is one of the quotients whose other neighbour is allowed."""
    m, _ = np.frexp(abs(b))
    q = Fraction(float(a)) / Fraction(float(b))
    mid = (Fraction(float(got)) + Fraction(float(want))) / 2
    return m > 1 - 2.0**-7 and got == np.nextafter(want, got) and abs(q - mid) <= abs(q) / 2**104
