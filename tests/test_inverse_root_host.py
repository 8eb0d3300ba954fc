"""The short FP64 inverse root (csrc/f64_math.cuh) in exact arithmetic: its two
corrections round every hard argument as the general square root and division do,
whichever double within 0.52 ulp of x^-1/2 they start from."""
from __future__ import annotations

from fractions import Fraction
from math import isqrt

import numpy as np
import pytest

from test_direct_gpu import _hard_arguments

Y_ULPS = Fraction(52, 100)


def _fma(a, b, c):
    return float(Fraction(a) * Fraction(b) + Fraction(c))  # rounded once, to nearest even


def _estimates(x):
    """The doubles within Y_ULPS of x^-1/2 (x an ordinary double)."""
    inverse = 1 / Fraction(x)
    scale = 1 << 400
    root = Fraction(isqrt(inverse.numerator * scale * scale // inverse.denominator), scale)
    nearest = float(root)
    out = []
    for y in (np.nextafter(nearest, 0.0), nearest, np.nextafter(nearest, np.inf)):
        ulp = Fraction(float(np.spacing(nearest)))
        if abs(Fraction(float(y)) - root) <= Y_ULPS * ulp + ulp / (1 << 200):
            out.append(float(y))
    return out


def _short(x, y):
    g = x * y
    s = _fma(_fma(-g, g, x), y / 2.0, g)
    return _fma(_fma(-s, y, 1.0), y, y)


def _covered(x):
    bits = int(np.float64(x).view(np.uint64))
    return 2.0 ** -895 <= x < 2.0 ** 897 and (bits & 0xffffffff) < 0xfffffffe


def test_every_hard_argument_rounds_as_the_general_operations_do():
    # One exponent of each parity stands for all: the steps scale exactly.
    arguments = sorted({float(x) for x in _hard_arguments() if 2.0 ** -60 < x < 2.0 ** 60})
    assert len(arguments) > 400
    tried = 0
    for x in arguments:
        if _covered(x):
            for y in _estimates(x):
                assert _short(x, y) == float(1.0 / np.sqrt(np.float64(x))), (x.hex(), y.hex())
                tried += 1
    assert tried > 400


@pytest.mark.parametrize("x", [4.0 - 2.0 ** -51, 4.0 - 2.0 ** -50])
def test_the_arguments_left_to_the_general_operations_need_them(x):
    assert not _covered(x) and not _covered(x * 4.0 ** 60)
    assert np.sqrt(x) == 2.0 - 2.0 ** -52
    assert any(_short(x, y) != 1.0 / np.sqrt(x) for y in (0.5, np.nextafter(0.5, 1.0)))
