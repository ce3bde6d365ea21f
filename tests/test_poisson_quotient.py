"""The smoother's quotient (tb_poisson.cu, relaxed): reciprocal, one Newton step and a correction by the
exact remainder give the correctly rounded FP32 quotient for every reciprocal within one ulp, here
in exact rational arithmetic.  Divisors with every mantissa bit set are the method's known
exception: one ulp.
"""
from fractions import Fraction

import numpy as np


def rn(v):
    """The FP32 number nearest to a rational of normal size, ties to even."""
    if v == 0:
        return Fraction(0)
    s, a = (-1, -v) if v < 0 else (1, v)
    e = a.numerator.bit_length() - a.denominator.bit_length() - 24
    scale = Fraction(2) ** e
    while a / scale >= 1 << 24:
        scale *= 2
    while a / scale < 1 << 23:
        scale /= 2
    q = a / scale
    n, rest = q.numerator // q.denominator, q - q.numerator // q.denominator
    if rest > Fraction(1, 2) or (rest == Fraction(1, 2) and n & 1):
        n += 1
    return s * n * scale


def test_quotient_is_correctly_rounded():
    rng = np.random.default_rng(4)
    s = np.concatenate([rng.normal(0, 1, 1500), rng.integers(1, 1 << 24, 1500)]).astype(np.float32)
    d = np.concatenate([rng.uniform(1e-3, 1e3, 1500), rng.integers(1, 1 << 24, 1500)]).astype(np.float32)
    s[:4], d[:4] = [1, 1, 16777215, 8388609], [3, 16777215, 8388609, 16777215]
    for a, b in zip(s, d):
        a, b = Fraction(float(a)), Fraction(float(b))
        y0 = np.float32(float(rn(1 / b)))
        for near in (np.nextafter(y0, np.float32(0)), y0, np.nextafter(y0, np.float32(np.inf))):
            y = Fraction(float(near))
            y = rn(y + y * rn(1 - b * y))
            q = rn(a * y)
            got, want = rn(q + y * rn(a - b * q)), rn(a / b)
            if np.float32(float(b)).view(np.uint32) & 0x7fffff == 0x7fffff:
                assert abs(got / want - 1) <= Fraction(1, 1 << 23)
            else:
                assert got == want
