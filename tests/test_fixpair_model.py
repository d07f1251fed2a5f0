"""The integer pair terms (dev_fixpair.cuh) restated with Python integers,
against exact rational arithmetic: positions on a 2^-61 grid, r^2 to 2^-57,
an FP32 rsqrt seed (up to 2^-22 off), series and products in 64-bit high
words, terms placed in a 128-bit sum. Bars, from the truncations: every step
stays inside its words; m/r within 2^-54 and each component of m d/r^3 within
2^-53 of the term (relative to the whole term, the components are aligned to
its largest)."""
import math
import random
from fractions import Fraction

import numpy as np

M32, M64 = 2**32 - 1, 2**64 - 1


def isqrt_frac(q, bits=140):
    """1/sqrt(q) to about 2^-bits relative, as a Fraction."""
    k = 2 * bits + max(0, q.numerator.bit_length() - q.denominator.bit_length())
    k += k & 1
    n = (q.denominator << (2 * k)) // q.numerator
    return Fraction(math.isqrt(n), 1 << k)


def mulhi(a, b):
    r = (a >> 32) * (b >> 32)
    r += ((a >> 32) * (b & M32)) >> 32
    r += ((a & M32) * (b >> 32)) >> 32
    assert r <= M64
    return r


def grid(xmax, eps):
    ex = math.frexp(max(xmax, eps))[1]
    g = 61 - ex
    E = int(math.ldexp(eps, g))
    assert E >= 1 << 48
    mant, e = math.frexp(eps * eps)
    S, k = int(mant * 2**53), e - 53
    return dict(g=g, eh=E >> 32, e2n=S << 9, e2s=64 + 9 - k - 2 * g)


def pair(f, d, rng):
    neg = [-1 if v < 0 else 0 for v in d]
    o = f["eh"]
    for v, g in zip(d, neg):
        o |= (v >> 32) ^ g
    s = 32 - o.bit_length() - 2
    assert 0 <= s <= 15
    n = [v << s for v in d]
    assert max(abs(v) for v in n) <= 1 << 62
    hh = sum((v >> 32) ** 2 for v in n)
    hl = sum((v >> 32) * ((v & M32) >> 2) for v in n)
    assert -(1 << 63) <= hl < 1 << 63
    sh = f["e2s"] - 2 * s
    assert sh >= 0
    r2 = hh + (hl >> 29) + (f["e2n"] >> sh) + 1
    assert 1 << 58 <= r2 <= (1 << 62) + 1
    h = r2 >> 32
    cut = max(0, h.bit_length() - 24)
    hf = (h >> cut) << cut
    y = np.float32((1.0 / math.sqrt(hf)) * (1 + rng.uniform(-1, 1) * 2**-22.4))
    yb = int(y.view(np.uint32))
    ey, Y = yb >> 23, ((yb << 8) | 0x80000000) & M32
    assert 111 <= ey <= 114
    S = Y * Y
    assert r2 << 1 <= M64
    T = mulhi(r2 << 1, S)
    k = 285 - 2 * ey
    e = (1 << k) - T
    assert -(1 << 63) <= e < 1 << 63
    e57 = e >> (k - 57)
    return n, neg, s, Y, ey, S, e57


def series(e57, num):
    eh = e57 >> 6
    assert -(1 << 31) <= eh < 1 << 31
    return ((((eh * eh) >> 36) & M32) * num) >> 12


def check(f, d, m, rng):
    em, mant = math.frexp(m)[1] + 1022, int(math.frexp(m)[0] * 2**53)
    ms = mant << 11
    n, neg, s, Y, ey, S, e57 = pair(f, d, rng)
    u = Fraction(1, 1) / Fraction(2) ** f["g"]
    eps2 = Fraction(f["e2n"]) * Fraction(2) ** (64 - f["e2s"]) * u * u
    r2 = sum(Fraction(v) ** 2 for v in d) * u * u + eps2
    ir = isqrt_frac(r2)
    # m / r
    c = (e57 >> 1) + series(e57, 3)
    C = (1 << 63) + (c << 6)
    assert 0 < C <= M64
    V = Y * (C >> 32) + ((Y * (C & M32)) >> 32)
    F = mulhi(V, ms)
    assert 1 << 60 <= F < 1 << 63
    X = ey + em + s + f["g"] - 1259
    got = Fraction(F) * Fraction(2) ** X
    want = Fraction(m) * ir
    assert abs(got / want - 1) <= Fraction(1, 2**54)
    # m d / r^3
    c = e57 + (e57 >> 1) + series(e57, 15)
    C = (1 << 63) + (c << 6)
    assert 0 < C <= M64
    W = Y * (S >> 32) + ((Y * (S & M32)) >> 32)
    assert W <= M64
    F = mulhi(mulhi(W, C), ms)
    assert F < 1 << 63
    X = 3 * ey + em + 2 * s + 2 * f["g"] - 1543
    w3 = Fraction(m) * ir**3 * u
    top = w3 * max(max(abs(v) for v in d), f["eh"] << 32)
    for v, nn in zip(d, n):
        P = mulhi(F, abs(nn))
        assert P < 1 << 61
        got = Fraction(P) * Fraction(2) ** X
        assert abs(got - w3 * abs(v)) <= top * Fraction(1, 2**53)


def test_pair_terms_against_rationals():
    rng = random.Random(11)
    for trial in range(4000):
        xmax = 2.0 ** rng.uniform(-20, 30)
        eps = xmax * 2.0 ** rng.uniform(-11.9, 1)
        mmax = 2.0 ** rng.uniform(-40, 40)
        f = grid(xmax, eps)
        lim = min(int(math.ldexp(xmax, f["g"])), (1 << 61) - 1)
        kind = rng.randrange(5)
        if kind == 0:  # anywhere
            d = [rng.randint(-2 * lim, 2 * lim) for _ in range(3)]
        elif kind == 1:  # close pairs
            b = rng.randrange(1, 61)
            d = [rng.randint(-(1 << b), 1 << b) for _ in range(3)]
        elif kind == 2:  # powers of two and their neighbours
            d = [rng.choice([-1, 1]) * ((1 << rng.randrange(0, 61)) + rng.randint(-1, 1))
                 for _ in range(3)]
        elif kind == 3:  # extremes
            d = [rng.choice([-2 * lim, 2 * lim, 0, lim, 1]) for _ in range(3)]
        else:
            d = [0, 0, 0]
        check(f, d, mmax * 2.0 ** -rng.uniform(0, 40), rng)


def test_sum_places_terms():
    """Fix128::add: (v 2^64) >> sh, negated for neg (less one unit), for every
    alignment, in 32-bit words."""
    rng = random.Random(5)
    for sh in list(range(0, 135)) + [160, 500]:
        for neg in (0, M32):
            v = rng.randrange(1 << 63)
            hi, lo = (v >> 32) ^ neg, (v & M32) ^ neg
            shi = hi - (1 << 32) if hi >> 31 else hi
            b, w = sh & 31, sh >> 5
            t2 = (shi >> b) & M32
            t1 = (((hi << 32) | lo) >> b) & M32
            t0 = (((lo << 32) | neg) >> b) & M32
            words = [neg] * 4
            for k, t in ((3 - w, t2), (2 - w, t1), (1 - w, t0)):
                if 0 <= k < 4:
                    words[k] = t
            got = sum(x << (32 * k) for k, x in enumerate(words))
            want = (v << 64) >> sh if sh < 128 else 0
            if neg:
                want = (-want - 1) % (1 << 128)
            assert got == want, (sh, neg)


def test_short_sum_places_terms():
    """Fix96::add: the 128-bit sum's term without its lowest word, cut downwards."""
    rng = random.Random(6)
    for sh in list(range(1, 100)) + [160, 500]:
        for neg in (0, M32):
            v = rng.randrange(1 << 63)
            x = ((v >> 32) ^ neg) << 32 | ((v & M32) ^ neg)
            sx = x - (1 << 64) if x >> 63 else x
            top = (sx >> min(sh, 63)) & M64
            low = ((x & M32) << (32 - sh)) & M32 if sh < 32 else (sx >> min(sh - 32, 63)) & M32
            got = top << 32 | low
            want = ((v << 32) >> sh) if not neg else ((-v - 1) << 32) >> sh
            slack = 0 if not neg or sh >= 32 else (1 << (32 - sh)) - 1
            assert 0 <= (got - want) % (1 << 96) <= slack, (sh, neg)
