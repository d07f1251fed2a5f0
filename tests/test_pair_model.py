"""The pair terms from FP64 differences (pair_r, pair_pack, pair_inv_r, pair_m_r3 in
dev_fixpair.cuh) restated with Python integers, against exact rational arithmetic:
every word stays in its range, 1/r and m/r^3 are within 1.1 x 2^-53 of the function of the
differences, for FP32 seeds 2^-22.4 off either way, differences of every relative
size, and the significands at the ends (terms just below and above powers of two)."""
import math
import random
import struct
from fractions import Fraction

import numpy as np

from test_fixpair_model import M32, M64, isqrt_frac

BAR = Fraction(11, 10) * Fraction(1, 2**53)


def bits(d):
    return struct.unpack("<Q", struct.pack("<d", d))[0]


def value(b):
    return struct.unpack("<d", struct.pack("<Q", b))[0]


def word(d, er):
    b = bits(d)
    h, l = b >> 32, b & M32
    top = (h & 0xFFFFF) | 0x100000
    v = ((top << 10 | l >> 22) & M32) << 32 | ((l << 10) & M32)
    return v >> min(er - (h >> 20 & 0x7FF), 64)


def eps_parts(eps):
    b = bits(eps * eps)
    eb = b >> 52
    if 0 < eb < 2047:
        return ((b & (2**52 - 1)) | 2**52) << 9, eb + 1022, bits(abs(eps)) >> 32
    assert eps == 0.0
    return 0, 0, 0


def pair(d, eps, off):
    e2n, e2s, eh = eps_parts(eps)
    er = max([bits(v) >> 32 & 0x7FFFFFFF for v in d] + [eh]) >> 20
    w = [word(v, er) for v in d]
    assert max(w) < 1 << 63
    hh = sum((v >> 32) ** 2 for v in w)
    hl = [(v >> 32) * (v & M32) for v in w]
    assert hl[0] + hl[1] <= M64
    sh = 2 * er - e2s
    assert sh >= 0
    r2 = hh + ((hl[0] + hl[1]) >> 31) + (hl[2] >> 31) + (e2n >> min(sh, 64)) + 2
    assert 1 << 60 <= r2 <= M64
    h = r2 >> 32
    cut = max(0, h.bit_length() - 24)
    y = np.float32((1.0 / math.sqrt((h >> cut) << cut)) * (1 + off))
    yb = int(y.view(np.uint32))
    ey, Y = yb >> 23, ((yb << 8) | 0x80000000) & M32
    assert 110 <= ey <= 113
    S = Y * Y
    T = (r2 * S) >> 64
    k = 284 - 2 * ey
    D = ((1 << k) - T) & M64  # in 64 bits
    D -= (D >> 63) << 64
    assert D == (1 << k) - T and abs(D) < 1 << (k - 20)
    return er, ey, Y, S, (D << 2) >> (k - 58)


def series(e60, num):
    """num / 8 e^2 2^60"""
    eh = e60 >> 9
    assert -(1 << 31) <= eh < 1 << 31
    return (((eh * eh) >> 36) * num) >> 9


def pack(F, E):
    assert 0 < F <= M64
    lz = 64 - F.bit_length()
    assert lz <= 5
    F = F << lz & M64
    hi, lo = F >> 32, F & M32
    E -= lz
    v = ((((E - 1) << 20) + (hi >> 11)) << 32) + (((hi << 32 | lo) >> 11) & M32)
    return value(v + (lo >> 10 & 1)), E


def inv_r(d, eps, off):
    er, ey, Y, S, e60 = pair(d, eps, off)
    C = (1 << 63) + (((e60 >> 1) + series(e60, 3)) << 3)
    V = Y * (C >> 32) + ((Y * (C & M32)) >> 32)
    v, E = pack(V, ey - er + 1934)
    assert er >= 65 and 1 <= E < 2046
    return v


def draws(rng, count):
    """Differences, eps and seed errors."""
    for t in range(count):
        scale = 2.0 ** rng.uniform(-60, 60)
        kind = rng.randrange(5)
        eps = rng.choice([0.0, scale * 2.0 ** rng.uniform(-70, 3)])
        if kind == 0:
            d = [scale * rng.uniform(-1, 1) for _ in range(3)]
        elif kind == 1:  # very different sizes
            d = [scale * rng.choice([-1, 1]) * 2.0 ** rng.uniform(-80, 0) for _ in range(3)]
        elif kind == 2:  # one axis, r at a power of two and beside it
            p = 2.0 ** rng.randrange(-60, 60) * (1 + rng.choice([0, 1, -1]) * 2.0 ** -rng.randrange(20, 53))
            d = [0.0, 0.0, 0.0]
            d[rng.randrange(3)] = p
            eps = rng.choice([0.0, p * 2.0 ** -40])
        elif kind == 3:  # all significand bits set, equal sizes
            p = scale * (2.0 - 2.0**-52)
            d = [p, -p, p]
            eps = rng.choice([0.0, p])
        else:  # softened only
            d, eps = [rng.choice([0.0, 1e-30 * scale]) for _ in range(3)], scale
        off = rng.choice([-1, 1, rng.uniform(-1, 1)]) * 2**-22.4
        yield [float(v) for v in d], float(eps), off


def r_squared(d, eps):
    return sum(Fraction(v) ** 2 for v in d) + Fraction(eps * eps)


def test_inverse_distance():
    rng = random.Random(3)
    for d, eps, off in draws(rng, 8000):
        want = isqrt_frac(r_squared(d, eps))
        assert abs(Fraction(inv_r(d, eps, off)) / want - 1) <= BAR, (d, eps, off)


def m_r3(d, eps, m, off):
    er, ey, Y, S, e60 = pair(d, eps, off)
    C = (1 << 63) + ((e60 + (e60 >> 1) + series(e60, 15)) << 3)
    assert 0 < C <= M64
    W = Y * (S >> 32) + ((Y * (S & M32)) >> 32)
    assert W <= M64
    b = bits(m)
    em, Mm = b >> 52, ((b & (2**52 - 1)) | 2**52) << 11
    v, E = pack((((W * C) >> 64) * Mm) >> 64, 3 * (ey - er) + em + 2734)
    assert er >= 65 and 1 <= em < 2047 and 1 <= E < 2046
    return v


def test_mass_over_distance_cubed():
    rng = random.Random(4)
    for d, eps, off in draws(rng, 8000):
        m = 2.0 ** rng.uniform(-200, 200)
        if rng.random() < 0.4:  # the ends of the significand
            m = 2.0 ** rng.randrange(-200, 200) * (1 + rng.choice([0.0, -(2.0**-53), 2.0**-52]))
        want = Fraction(m) * isqrt_frac(r_squared(d, eps)) ** 3
        assert abs(Fraction(m_r3(d, eps, m, off)) / want - 1) <= BAR, (d, eps, m, off)
