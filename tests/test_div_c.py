"""Division by the speed of light as x zh + RN(x zl) (Brisebarre, Muller & Raina
2004), as the resolve of a tree's children computes it: correctly rounded on
random quotients and on those nearest to a midpoint of two doubles."""

from __future__ import annotations

import ctypes
import ctypes.util
from fractions import Fraction

import numpy as np
import pytest

C = 299792458
ZH = float.fromhex("0x1.ca726eb25f9dbp-29")
ZL = float.fromhex("0x1.568bbb3de4666p-84")


def _hard_cases():
    """x whose quotients lie next to midpoints: (2k + 1) C / 2^e rounded both ways."""
    rng = np.random.default_rng(3)
    out = []
    for k in rng.integers(1 << 52, 1 << 53, 400).tolist():
        mid = Fraction(2 * k + 1, 1 << 53) * C
        x = float(mid)
        out += [x, np.nextafter(x, np.inf), np.nextafter(x, -np.inf)]
    return [float(v) for v in out]


@pytest.mark.parametrize("scale", [-820, -300, -30, 0, 40, 300, 740])
@pytest.mark.parametrize("sign", [1.0, -1.0])
def test_division_by_c_is_correctly_rounded(scale, sign):
    libm = ctypes.CDLL(ctypes.util.find_library("m"))
    libm.fma.restype = ctypes.c_double
    libm.fma.argtypes = [ctypes.c_double] * 3
    assert ZH == 1.0 / C
    assert float(Fraction(1, C) - Fraction(ZH)) == ZL
    rng = np.random.default_rng(scale + 1000)
    xs = [float(v) for v in rng.uniform(1, 2, 400)] + _hard_cases()
    for v in xs:
        x = sign * np.ldexp(v, scale)
        x = float(x)
        assert libm.fma(x, ZH, x * ZL) == x / C
