"""CPU model of the Gram's slice products as k_zone_gram_oz forms them (zone_gram_oz.cu,
oz_slices.cuh): the integer steps in Python integers and NumPy, against exact arithmetic.

* fixed_row: the upper 64 bits of the significands' product shifted to the fixed point once, within
  half a unit and 2^-9 of one (the truncated bits) of the exact value at every shift; products of
  2^56 units on and non-finite factors are flagged, zero and subnormal ones give 0.
* stage_digits flags every value that seven digits do not hold, and no other.
* digit_pairs: the FP16 numbers 0x6400 | byte less 1152 are the balanced base-256 digits.
* The Gram over several accumulator reads: levels 0..7, even and odd first digits apart, levels 0..3
  and 4..7 (level 7 rounded to units of level 6 at each read of each half) as 64-bit integers, added
  and scaled to FP64 at the end; its error is the rounding of X, the dropped levels 8 to 12, the
  roundings of level 7 and two of FP64.
* fixed_of and scaled_i64: conversion to fixed point and back over FP64's whole range, subnormal
  numbers included.
"""
import math
import struct
from fractions import Fraction

import numpy as np

M64 = (1 << 64) - 1
BIAS = 0x80808080808080


def _bits(x):
    return struct.unpack("<Q", struct.pack("<d", float(x)))[0]


def _float(b):
    return struct.unpack("<d", struct.pack("<Q", b))[0]


def fixed_row(m, es, h, E):
    """The kernel's steps (64-bit words); None where it sets its bad flag."""
    hb = _bits(h)
    eh = (hb >> 52) & 0x7FF
    mh = ((hb & 0xFFFFFFFFFFFFF) | 0x10000000000000) << 10
    r = 2053 + E - es - eh
    if eh == 0x7FF or (r < 7 and m != 0 and eh != 0):
        return None
    top = (m * mh) >> 64
    F = ((top + (1 << (r - 1))) & M64) >> r if (r < 64 and eh != 0) else 0
    return -F if hb >> 63 else F


def weight_parts(s):
    """What the kernel keeps of |w| / sqrt(r): the significand << 11 and the biased exponent."""
    sb = _bits(s)
    es = (sb >> 52) & 0x7FF
    return (((sb & 0xFFFFFFFFFFFFF) | 0x10000000000000) << 11 if es else 0), es


def digits(F):
    U = (F + BIAS) & M64
    return [((U >> (8 * (6 - p))) & 255) - 128 for p in range(7)]


def test_fixed_row_rounds_once_at_every_shift():
    rng = np.random.default_rng(3)
    seen = set()
    for _ in range(20000):
        s = float(rng.uniform(1, 2)) * 2.0 ** int(rng.integers(-40, 3))
        h = float(rng.uniform(-2, 2)) * 2.0 ** int(rng.integers(-40, 30))
        E = int(rng.integers(-60, 60))
        if rng.random() < 0.3:  # near the bound
            E = math.frexp(s * h)[1] + int(rng.integers(-2, 2))
        m, es = weight_parts(s)
        F = fixed_row(m, es, h, E)
        exact = Fraction(s) * Fraction(h) * Fraction(2) ** (54 - E)
        r = 2053 + E - es - ((_bits(h) >> 52) & 0x7FF)
        seen.add(r)
        if F is None:
            assert abs(exact) >= 1 << 55
        else:
            assert abs(F) <= 1 << 56 and abs(F - exact) <= Fraction(1, 2) + Fraction(1, 512)
    assert {5, 6, 7, 8, 9, 62, 63, 64, 65} <= seen


def test_fixed_row_flags_and_zeros():
    m, es = weight_parts(1.0)
    assert fixed_row(m, es, 1.0, 0) == 1 << 54
    assert fixed_row(m, es, math.nextafter(1.0, 2.0), 0) == (1 << 54) + 4
    m2, es2 = weight_parts(1.5)
    assert fixed_row(m2, es2, 1.5, 0) == 9 << 52  # r = 7, 2.25 times the bound
    assert fixed_row(m, es, 2.0, 0) is None       # r = 6
    assert fixed_row(m, es, float("inf"), 0) is None and fixed_row(m, es, float("nan"), 0) is None
    assert fixed_row(*weight_parts(0.0), 1e300, 0) == 0
    assert fixed_row(m, es, 0.0, 0) == 0 and fixed_row(m, es, 5e-324, -1074 + 40) == 0


def test_digit_pairs_are_fp16_digits():
    byte = np.arange(256, dtype=np.uint16)
    h = (byte | np.uint16(0x6400)).view(np.float16) - np.uint16(0x6480).view(np.float16)
    assert np.array_equal(h.astype(int), byte.astype(int) - 128)


def test_staged_digits_hold_the_value_or_flag_it():
    edge = 0x7F7F7F7F7F7F7F  # seven digits of 127
    rng = np.random.default_rng(6)
    near = [s * (e + k) for s in (1, -1) for e in (edge, BIAS, 1 << 54, 1 << 55, 1 << 56) for k in
            range(-3, 4)]
    for F in near + [int(x) for x in rng.integers(-(1 << 57), 1 << 57, 3000)] + [0, 1 << 54]:
        value = sum(d * 256 ** (6 - p) for p, d in enumerate(digits(F)))
        held = ((F + BIAS) & M64) >> 56 == 0
        assert held == (value == F)
        assert held == (-BIAS <= F <= edge)


def _halves(F, p_set, level):
    """sum over p in p_set, p + q = level of D_p^T D_q for rows F (k, N); FP32 sums stay exact."""
    D = np.array([[digits(int(f)) for f in row] for row in F]).transpose(2, 0, 1)  # (7, k, N)
    out = np.zeros((F.shape[1],) * 2, dtype=object)
    for p in p_set:
        q = level - p
        if 0 <= q <= 6 and p <= 6:
            out = out + (D[p].T @ D[q]).astype(object)
    assert np.abs(out.astype(float)).max() <= 2 ** 24
    return out


def scaled(v, e2):
    """scaled_i64: v 2^e2 rounded to nearest even."""
    if v == 0:
        return 0.0
    sgn, m = (1 << 63 if v < 0 else 0), abs(v)
    lz = 64 - m.bit_length()
    be = 63 - lz + e2 + 1023
    mm = (m << lz) & M64
    if be < 1:
        sh = 12 - be
        if sh > 64:
            return _float(sgn)
        q = mm >> sh if sh < 64 else 0
        rem = (mm << (64 - sh)) & M64 if sh < 64 else mm
        return _float(sgn | (q + (1 if rem > 1 << 63 or (rem == 1 << 63 and q & 1) else 0)))
    if be > 2046:
        return _float(sgn | 0x7FF0000000000000)
    mant, rem = (mm >> 11) & 0xFFFFFFFFFFFFF, mm & 0x7FF
    return _float(sgn | ((be << 52) + mant + (1 if rem > 0x400 or (rem == 0x400 and mant & 1) else 0)))


def fixed_of(x, B, E):
    """round(x 2^(B - E)) for |x| < 2^E."""
    b = _bits(x)
    e = (b >> 52) & 0x7FF
    m = (b & 0xFFFFFFFFFFFFF) | 0x10000000000000
    if e == 0:
        m ^= 0x10000000000000
        e = 1
    s = e - 1075 + B - E
    F = m << min(s, 10) if s >= 0 else ((m + (1 << (-s - 1))) >> -s if s > -55 else 0)
    return -F if b >> 63 else F


def test_gram_over_several_reads():
    rng = np.random.default_rng(8)
    N, p = 5, 700  # three reads of 256 observations
    h = rng.standard_normal((p, N)) * 10.0 ** np.array([0, -3, 2, 0, -1])
    s = rng.uniform(0.01, 1.0, p) * np.exp(-rng.uniform(0, 9, p))
    E = [math.frexp(float(np.abs(h[:, a] * s).max()) * (1 + 2.0 ** -20))[1] for a in range(N)]
    parts = [weight_parts(x) for x in s]
    F = np.array([[fixed_row(*parts[q], h[q, a], E[a]) for a in range(N)] for q in range(p)],
                 dtype=object)
    hi = np.zeros((N, N), dtype=object)
    lo = np.zeros((N, N), dtype=object)
    reads = 0
    for k0 in range(0, p, 256):
        rows = F[k0:k0 + 256]
        reads += 1
        for odd in (0, 1):
            lev = [_halves(rows, range(odd, 7, 2), L) for L in range(8)]
            hi = hi + lev[0] * 2 ** 24 + lev[1] * 2 ** 16 + lev[2] * 2 ** 8 + lev[3]
            lo = lo + lev[4] * 2 ** 16 + lev[5] * 2 ** 8 + lev[6] + (lev[7] + 128) // 256
    X = [[Fraction(float(h[q, a])) * Fraction(float(s[q])) for a in range(N)] for q in range(p)]
    for a in range(N):
        for b in range(a + 1):
            ex = E[a] + E[b]
            got = scaled(int(hi[a, b]), ex - 36) + scaled(int(lo[a, b]), ex - 60)
            exact = sum(X[q][a] * X[q][b] for q in range(p))
            unit = Fraction(2) ** ex
            bound = (sum(abs(X[q][a]) * Fraction(2) ** E[b] + abs(X[q][b]) * Fraction(2) ** E[a]
                         for q in range(p)) * Fraction(257, 512) / 2 ** 54      # X's fixed point
                     + p * unit / 2 ** 59                                       # levels 8 to 12
                     + 2 * reads * unit / 2 ** 60                               # level 7, half a unit
                     + 3 * abs(exact) / 2 ** 53)                                # FP64
            assert abs(Fraction(got) - exact) <= bound


def test_fixed_point_over_the_whole_range():
    rng = np.random.default_rng(5)
    for _ in range(5000):
        e = int(rng.integers(-1074, 1000))
        E = e + int(rng.integers(1, 60))
        if E < -1022:
            E = -1022
        x = math.ldexp(float(rng.uniform(-1, 1)), e)
        exact = Fraction(x) * Fraction(2) ** (54 - E)
        F = fixed_of(x, 54, E)
        assert abs(F - exact) <= Fraction(1, 2)
        if abs(x) < 2.0 ** -1022:  # subnormal numbers below the smallest bound are exact
            assert E > -1020 or F == exact
    for _ in range(20000):
        bits = int(rng.integers(1, 64))
        v = (int(rng.integers(0, 1 << 62)) << 1 | int(rng.integers(0, 2))) >> (63 - bits) | 1 << (bits - 1)
        if rng.random() < 0.3 and bits > 12:  # ties
            v = (1 << (bits - 1)) | (int(rng.integers(0, 8)) << max(0, bits - 56))
        v = -v if rng.random() < 0.5 else v
        e2 = int(rng.choice([rng.integers(-1150, -1000), rng.integers(900, 1030), rng.integers(-60, 60)]))
        f = Fraction(v) * Fraction(2) ** e2
        try:
            exact = f.numerator / f.denominator  # correctly rounded
        except OverflowError:
            exact = math.copysign(math.inf, v)
        assert scaled(v, e2) == exact
