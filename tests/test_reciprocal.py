"""rcp64 of flash-x_b200/csrc/fxb_device.cuh: three Newton-Raphson steps on a
hardware approximation of 1/b return the correctly rounded reciprocal for
every b whose significand is not all ones (that one takes the division
operator).  Restated here with exact rational fused multiply-adds, from
approximations down to 2^-20 relative; the device parity tests then compare
whole steps bit for bit."""
import random
import struct
from fractions import Fraction

import pytest


def _fma(a, b, c):
    return float(Fraction(a) * Fraction(b) + Fraction(c))


def _rcp64(b, rel):
    y = float(Fraction(1) / Fraction(b) * (1 + Fraction(rel)))
    y = struct.unpack("<d", struct.pack("<Q", struct.unpack("<Q", struct.pack("<d", y))[0] & ~0xFFFFFFFF))[0]
    for _ in range(3):
        y = _fma(y, _fma(-b, y, 1.0), y)
    return y


def _make(exp, mant, sign=0):
    return struct.unpack("<d", struct.pack("<Q", (sign << 63) | ((1023 + exp) << 52) | mant))[0]


@pytest.mark.parametrize("rel", [0.0, 2.0 ** -20, -2.0 ** -20, 2.0 ** -23])
def test_reciprocal_is_correctly_rounded(rel):
    rng = random.Random(20261204)
    ones = (1 << 52) - 1
    mants = [0, 1, 2, 3, ones - 1, ones - 2, ones - 3, 1 << 51, (1 << 51) - 1, (1 << 51) + 1]
    mants += [ones - rng.getrandbits(20) - 1 for _ in range(800)] + [rng.getrandbits(20) for _ in range(800)]
    mants += [rng.getrandbits(52) for _ in range(3000)]
    bad = []
    for m in mants:
        b = _make(rng.randint(-400, 399), m, rng.getrandbits(1))
        if _rcp64(b, rel) != 1.0 / b:
            bad.append(b)
    assert not bad, f"{len(bad)} reciprocals differ from 1 / b, first b = {bad[0]!r}"
