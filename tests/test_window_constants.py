"""The two short forms of a division in the window loops (cvt_b200/csrc/pm_window.cuh), with the constants read from
the source: a colour byte / 255 in one fma, and x / 0.05 as a two-term product.  Exact arithmetic on the CPU."""
import os
import re
from fractions import Fraction

import numpy as np

from conftest import ROOT


def constant(name):
    src = open(os.path.join(ROOT, "cvt_b200", "csrc", "pm_window.cuh")).read()
    text = re.search(r"#define %s (\S+)f\b" % name, src).group(1)
    return float.fromhex(text) if text.startswith("0x") else float(np.float32(text))


def nearest_float(q):
    """the positive Fraction q rounded to a normal float, ties to even"""
    e = 0
    while q >= 2 ** (e + 1):
        e += 1
    while q < Fraction(2) ** e:
        e -= 1
    scaled = q / Fraction(2) ** (e - 23)   # in [2^23, 2^24)
    n = int(scaled)
    rest = scaled - n
    if rest > Fraction(1, 2) or (rest == Fraction(1, 2) and n % 2):
        n += 1
    return Fraction(n) * Fraction(2) ** (e - 23)


def test_colour_byte_over_255_for_every_byte():
    """pair_unit: fma(x, PM_RGB, x) for x = 257 byte 2^-141 is byte / 255 correctly rounded"""
    rgb = Fraction(constant("PM_RGB"))
    for byte in range(1, 256):
        bits = byte << 8 | byte << 16   # the byte twice, in bits 8-23: a float of exponent field 0 or 1
        x = Fraction(float(np.array([bits], np.uint32).view(np.float32)[0]))
        assert x == Fraction(257 * byte, 2 ** 141)
        assert nearest_float(x * rgb + x) == nearest_float(Fraction(byte, 255)), byte
        assert float(np.float32(byte) / np.float32(255)) == float(nearest_float(Fraction(byte, 255)))


def test_division_by_five_hundredths():
    """trunc_ad: fma(x, 20, x PM_D005) is x / 0.05f correctly rounded for every float from 2^-100 to 0.05f.  Both sides
    scale by powers of two while nothing underflows, so every mantissa is taken in the lowest, a middle and the
    highest full binade, and in the part of the next up to 0.05f.  20 x + RN(x D005) has at most 51 bits: a
    double holds it."""
    d005, c = np.float32(constant("PM_D005")), np.float32(0.05)
    m = np.arange(2 ** 23, dtype=np.uint32)
    for e in (-100, -40, -6, -5):
        x = (m | np.uint32((127 + e) << 23)).view(np.float32)
        x = x[x <= c]
        assert x.size == 2 ** 23 or e == -5
        small = (x.astype(np.float64) * np.float64(d005)).astype(np.float32)   # 48 bits: one rounding
        got = (x.astype(np.float64) * 20.0 + small.astype(np.float64)).astype(np.float32)
        assert (got == x / c).all(), e
    assert np.float32(0.0) * np.float32(20.0) + np.float32(0.0) * d005 == np.float32(0.0) / c
