"""CPU restatement of the words that FP64 stages hold their stencil inputs in
(hpc-reading-course_gb300/csrc/wave2d_fixed.cuh: fx_pack, fx_unpack, fx_least, fx_sum), checked
with exact rational arithmetic: a word gives its double back exactly, values that have none are
marked, and a stencil's error is bounded by the largest value that it reads itself.
"""
from fractions import Fraction

import numpy as np
import pytest

from test_fixed_point_arithmetic import COEF, DEN, WEIGHTS, bits, from_bits
from test_fixed_point_kinds import fx_to

TOP, NONE = 1087, 1023


def pack(v):
    """(word, has none)"""
    b = bits(v)
    if not b & (2 ** 63 - 1):
        return NONE, False
    r = (TOP - ((b >> 52) & 0x7FF)) & 0xFFFFFFFF
    m = ((b & (2 ** 52 - 1)) | 2 ** 52) << 10
    return ((-m if b >> 63 else m) | (r & 1023)), r >= NONE


def unpack(w):
    r, m = w & 1023, w & ~1023
    a = abs(m)
    if a == 0:
        return 0.0
    hw = ((TOP - r - 1) << 20) + (a >> 42)
    return from_bits(((hw | (0x80000000 if w < 0 else 0)) << 32) | ((a >> 10) & 0xFFFFFFFF))


def least(words, R):
    return min([NONE] + [words[R + k] & 1023 for k in range(-R, R + 1) if k])


def stencil(words, order, r):
    R = order // 2
    at = [0 if k == R else (w & ~1023) >> min(64, (w & 1023) - r + 8) for k, w in enumerate(words)]
    return sum(c * (at[R + k + 1] - at[R - k - 1]) for k, c in enumerate(WEIGHTS[order]))


def _values(rng, n, lo=-950, hi=63):
    return (rng.choice([-1.0, 1.0], n) * rng.uniform(1.0, 2.0, n) * 2.0 ** rng.integers(lo, hi, n)).tolist()


def test_words_are_exact():
    rng = np.random.default_rng(0)
    edge = [2.0 ** -958, -(2.0 ** -958), np.nextafter(2.0 ** 65, 0), -np.nextafter(2.0 ** 65, 0), 1.0, -1.0, 0.0]
    for v in _values(rng, 3000) + edge:
        w, none = pack(float(v))
        assert not none and -(2 ** 63) <= w < 2 ** 63
        assert unpack(w) == v


def test_values_without_a_word_are_marked():
    for v in (2.0 ** 65, -(2.0 ** 65), 1e300, np.inf, -np.inf, np.nan, np.nextafter(2.0 ** -958, 0), 1e-300, 5e-324,
              -1e-310):
        assert pack(float(v))[1]
    assert pack(-0.0) == (NONE, False) and unpack(NONE) == 0.0


@pytest.mark.parametrize("order", [2, 4, 6])
def test_a_stencil_errs_by_its_own_largest_value(order):
    R = order // 2
    rng = np.random.default_rng(order)
    weight = 2 * sum(abs(c) for c in WEIGHTS[order])
    for trial in range(1500):
        e0 = int(rng.integers(-900, 60))
        line = _values(rng, 2 * R + 1, max(-957, e0 - int(rng.integers(1, 90))), e0 + 1)
        if trial % 3 == 0:
            line[int(rng.integers(0, 2 * R + 1))] = 0.0
        words = [pack(v)[0] for v in line]
        r = least(words, R)
        s = stencil(words, order, r)
        assert abs(2 * s) < 2 ** 63  # two such sums together stay in range
        exact = DEN[order] * sum(c * Fraction(v) for c, v in zip(COEF[order], line))
        unit = Fraction(2) ** (TOP - r - 1077)  # 2^-54 of the largest value's binade
        got = Fraction(fx_to(s, TOP - r))
        assert abs(got - exact) <= weight * unit + abs(got) * Fraction(1, 2 ** 53)
        big = max(abs(Fraction(line[R + k])) for k in range(-R, R + 1) if k)
        assert unit <= big * Fraction(1, 2 ** 54)


def test_zeros_and_far_smaller_values():
    zero = pack(0.0)[0]
    assert least([zero] * 5, 2) == NONE and stencil([zero] * 5, 4, NONE) == 0
    words = [pack(v)[0] for v in (1e-200, 0.0, 3.0, -1.0, -1e-250)]
    r = least(words, 2)
    # a shift that takes every bit leaves 0 or, below zero, -1 unit
    assert abs(Fraction(fx_to(stencil(words, 4, r), TOP - r)) + 8) <= Fraction(2) ** (TOP - r - 1077)
