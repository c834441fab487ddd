"""The integer series behind the rational rotations (turn_cos_sin): its
coefficients are the Taylor coefficients of sin(pi/4 u) / u and cos(pi/4 u) in
u^2, and a restatement of its steps in exact integers stays within 2^-59 of
the values before the one rounding to double.

The bound, in units of 2^-64 of the cosine: u^2 is cut below 2^-62 (4 units at
a derivative below 0.31); each of six steps cuts up to 2 and its coefficient
is off by up to 1, and with alternating signs the worst sum is 11; the last bit
cut when the value is handed over is 2. 13 on values of at least 0.707 are
below 19 relative, and the sine's steps are half as coarse.
"""
from __future__ import annotations

import math
import random
import re
from decimal import Decimal, localcontext
from pathlib import Path

import pytest

SOURCE = Path(__file__).resolve().parent.parent / "sparqsim_gb300" / "csrc" / "group_ops.cu"
PI = Decimal("3.14159265358979323846264338327950288419716939937510582097494459230781640628620899")
M64, M32 = (1 << 64) - 1, (1 << 32) - 1


def _coefficient(k, scale):
    with localcontext() as ctx:
        ctx.prec = 60
        return int(((PI / 4) ** k / math.factorial(k) * (1 << scale)).to_integral_value())


SIN64 = [_coefficient(2 * i + 1, 64) for i in range(6)]
SIN68 = [_coefficient(2 * i + 1, 68) for i in range(6, 10)]
COS63 = [_coefficient(2 * i, 63) for i in range(6)]
COS64 = [_coefficient(2 * i, 64) for i in range(6, 10)]


@pytest.mark.parametrize("name,want", [("kSin64", SIN64), ("kSin68", SIN68), ("kCos63", COS63), ("kCos64", COS64)])
def test_coefficients(name, want):
    body = re.search(name + r"\[\d\] = \{([^}]*)\}", SOURCE.read_text()).group(1)
    assert [int(x.strip().rstrip("ul"), 16) for x in body.split(",")] == want


def _series(u):
    """(sin, cos) of pi/4 u / 2^61 as exact fractions (numerator, exponent of 2)."""
    t = min(((u << 2) * (u << 2)) >> 64, (1 << 62) - 1)
    T = t << 2
    T32 = T >> 32
    s32, c32 = SIN68[3], COS64[3]
    for k in (2, 1, 0):
        s32 = (SIN68[k] - (s32 * T32 >> 32)) & M32
        c32 = (COS64[k] - (c32 * T32 >> 32)) & M32
    s, c = s32 >> 4, c32 >> 1
    for k in (5, 4, 3, 2, 1, 0):
        s = (SIN64[k] - (s * T >> 64)) & M64
        c = (COS63[k] - (c * T >> 64)) & M64
    lz = 64 - u.bit_length() if u else 0
    ym = (((u << lz) * s) >> 64) >> 1
    return (ym, 60 + lz), (c >> 1, 62)


def _exact(u):
    x = PI / 4 * Decimal(u) / Decimal(1 << 61)
    s, c, t = Decimal(0), Decimal(0), Decimal(1)
    for k in range(0, 44, 2):
        c += t
        t = t * x / (k + 1)
        s += t
        t = -t * x / (k + 2)
    return s, c


def test_series_error():
    rng = random.Random(5)
    us = [1, 2, 3, (1 << 61) - 1, 1 << 61, 0x1FDA22CCE1E97984]
    us += [rng.randrange(1, (1 << 61) + 1) for _ in range(2500)]
    us += [(1 << 61) - rng.randrange(1, 1 << 58) for _ in range(1500)]
    us += [rng.randrange(1 << b, 2 << b) for b in range(60) for _ in range(5)]
    with localcontext() as ctx:
        ctx.prec = 45
        for u in us:
            for (num, e), want in zip(_series(u), _exact(u)):
                assert abs(Decimal(num) / Decimal(1 << e) / want - 1) < Decimal(2) ** -59
