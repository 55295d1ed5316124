"""The float identities of the tracking passes: square roots compared with a
constant replaced by a comparison of the radicand with the largest float whose
correctly rounded root passes, and a Sobel value / 9 by one reciprocal and
Markstein's correction step."""
from fractions import Fraction

import numpy as np


def test_root_thresholds():
    for bits, c, strict in ((0x3c23d70b, 0.1, False), (0x3c23d709, 0.1, True), (0x3eb851eb, 0.6, True)):
        x = np.arange(bits - (1 << 18), bits + (1 << 18), dtype=np.uint32).view(np.float32)
        root = np.sqrt(x)   # correctly rounded in binary32
        want = root < np.float32(c) if strict else root <= np.float32(c)
        got = x <= np.uint32(bits).view(np.float32)
        assert np.array_equal(want, got), (hex(bits), c)


def _rn(q):
    """Fraction -> nearest binary32 (ties to even), as a Fraction; normal range or zero."""
    if q == 0:
        return q
    e = 0
    while abs(q) >= 2:
        q, e = q / 2, e + 1
    while abs(q) < 1:
        q, e = q * 2, e - 1
    n = q * (1 << 23)
    f = n.numerator // n.denominator
    r = n - f
    if r > Fraction(1, 2) or (r == Fraction(1, 2) and f & 1):
        f += 1
    return Fraction(f, 1 << 23) * Fraction(2) ** e


def test_sobel_ninth():
    y = Fraction(float(np.uint32(0x3de38e39).view(np.float32)))
    assert y == _rn(Fraction(1, 9))
    for d in range(-1020, 1021):
        q = _rn(d * y)
        r = _rn(d - 9 * q)
        got = q if r == 0 else _rn(r * y + q)
        assert got == _rn(Fraction(d, 9)), d
