"""CPU check of the signed bucket map for doubles (BucketMap<double> in hpdex_gb300/csrc/mwu_rank.cuh), which
works on the bits alone: floor(|x| * 2^(52 - E0)) below 2^E0 is the mantissa shifted right. The
C++ expression is restated in Python integers and compared with the definition in exact rational
arithmetic; the map has to be non-decreasing and to stay inside the bucket table (a value
outside it would index shared memory out of range): normals of every exponent, subnormals, signed zeros, the
values next to the junction, infinite-magnitude neighbours."""
import struct
from fractions import Fraction

import numpy as np

M64 = (1 << 64) - 1


def bits(x):
    return struct.unpack("<Q", struct.pack("<d", x))[0]


def key(x):
    u = bits(x)
    if (u << 1) & M64 == 0:
        u = 0
    return u ^ M64 if u >> 63 else u | 1 << 63


def e0_of(lo, hi):
    """max(ea - 12, -960), ea the exponent field of the smaller extreme magnitude, less 1022"""
    return max((bits(min(abs(lo), abs(hi))) >> 52 & 0x7FF) - 1022 - 12, -960)


def m_of(k, e0):
    """the kernel's integer form"""
    negative = not k >> 63
    b = (k ^ M64 if negative else k) & (M64 >> 1)
    b0 = (e0 + 1023) << 52
    ex = b >> 52
    sh = e0 + 1023 - (ex if ex else 1)
    mant = b & ((1 << 52) - 1) | (1 << 52 if ex else 0)
    u = b - b0 + (1 << 52) if b >= b0 else mant >> sh if sh < 64 else 0
    assert b >= b0 or sh >= 0
    return ((1 << 63) - u if negative else (1 << 63) + u) & M64


def defined(x, e0):
    t = abs(Fraction(x))
    if t < Fraction(2) ** e0:
        u = int(t * Fraction(2) ** (52 - e0))
    else:
        u = bits(abs(x)) - ((e0 + 1023) << 52) + (1 << 52)
    return (1 << 63) - u if x < 0 else (1 << 63) + u


def _values(rng, trial):
    scale = 2.0 ** rng.uniform(-1060, 1010)
    with np.errstate(over="ignore", under="ignore"):
        v = rng.standard_normal(400) * scale * 2.0 ** rng.uniform(-30, 10, 400)
    v = np.concatenate([v, np.ldexp(rng.uniform(-1, 1, 200), rng.integers(-1074, 1024, 200)) if trial % 2 else v,
                        [-0.0, 0.0, 5e-324, -5e-324, 2.2250738585072014e-308, -2.225073858507201e-308]])
    return v[np.isfinite(v)]


def test_integer_form_equals_the_definition_and_stays_in_the_table():
    rng = np.random.default_rng(2)
    for trial in range(120):
        v = _values(rng, trial)
        lo, hi = float(v.min()), float(v.max())
        if not lo < 0 < hi:
            continue
        e0 = e0_of(lo, hi)
        j = 2.0 ** e0
        edge = [s * x for x in (j, np.nextafter(j, 0), np.nextafter(j, np.inf), j / 2, 2 * j) for s in (1, -1)]
        v = sorted([float(x) for x in v] + [float(x) for x in edge if lo <= x <= hi])
        m = [m_of(key(x), e0) for x in v]
        assert m == [defined(x, e0) for x in v], trial
        base, top = m[0], m[-1]
        for nbl in (9, 11, 13):
            shift = max(0, (top - base).bit_length() - nbl)
            b = [(x - base) >> shift for x in m]
            assert all(x <= y for x, y in zip(b, b[1:])), trial
            assert b[0] == 0 and b[-1] < 1 << nbl, trial


def test_the_smallest_junction():
    """E0 at its floor (the extremes are subnormal or tiny) and at the top of the exponents"""
    for lo, hi in ((-5e-324, 5e-324), (-1e-300, 1e-290), (-1.7e308, 1.7e308), (-5e-324, 1.7e308)):
        e0 = e0_of(lo, hi)
        assert -960 <= e0 <= 1012
        v = sorted([lo, hi, 0.0, lo / 2, hi / 2, -5e-324, 5e-324, hi / 3e5])
        m = [m_of(key(x), e0) for x in v]
        assert m == [defined(x, e0) for x in v]
        assert all(x <= y for x, y in zip(m, m[1:]))
