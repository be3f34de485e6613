"""CPU model of the line transforms' integer arithmetic (csrc/bfp.cuh), in
Python integers: the twiddle product from signed 32-bit limbs without the low
limbs' product, the product by 1/sqrt(2), and the conversions from and to double.

A component of a product is two factors' h h' 2^64 + (h l' + l h') 2^32 + l l',
over 2^62, rounded once.  The two l l' terms left out are at most 2^31 2^31 /
2^62 = 1 unit each, so the error is below 1/2 + 2 units; every 64-bit
intermediate has to stay in range for complex magnitudes up to 2^62.
"""
import math
import random
from fractions import Fraction

import pytest

TOP = 62


def chk(v):
    assert -(1 << 63) <= v < (1 << 63), "64-bit overflow"
    return v


def limbs(v):
    lo = ((v + (1 << 31)) & 0xFFFFFFFF) - (1 << 31)
    hi = (v - lo) >> 32
    assert -(1 << 31) <= hi < (1 << 31)
    return hi, lo


def twiddle(angle):
    def one(v):
        hi, lo = limbs(round(Fraction(v) * 2 ** TOP))
        return hi, (lo if lo != -(1 << 31) else lo + 1)
    return one(math.cos(angle)) + one(math.sin(angle))


def cmul(X, Y, w, conj):
    xh, xl = limbs(X)
    yh, yl = limbs(Y)
    rz, rw, iz, iw = (w[2], w[3], -w[2], -w[3]) if conj else (-w[2], -w[3], w[2], w[3])
    out = []
    for a, al, p, pl, b, bl, q, ql in ((xh, xl, w[0], w[1], yh, yl, rz, rw), (yh, yl, w[0], w[1], xh, xl, iz, iw)):
        h = chk(a * p + b * q)
        m = 1 << 29
        for t in (a * pl, al * p, b * ql, bl * q):
            m = chk(m + t)
        out.append(chk(4 * h + (m >> 30)))
    return out


@pytest.mark.parametrize("conj", [False, True])
@pytest.mark.parametrize("bits", [3, 31, 33, 61])
def test_product_error_and_range(conj, bits):
    rng = random.Random(bits + 7 * conj)
    angles = [0.0, math.pi / 2, math.pi, -math.pi / 2, math.pi / 4] + [rng.uniform(-4, 4) for _ in range(200)]
    for a in angles:
        w = twiddle(a)
        W = [(w[0] << 32) + w[1], (w[2] << 32) + w[3]]
        for _ in range(20):
            r, t = 2.0 ** bits * rng.uniform(0.5, 2.0), rng.uniform(0, 7)   # magnitudes up to 2^62
            X, Y = int(r * math.cos(t)), int(r * math.sin(t))
            s = -1 if conj else 1
            want = (X * W[0] - s * Y * W[1], Y * W[0] + s * X * W[1])
            for g, e in zip(cmul(X, Y, w, conj), want):
                assert abs(Fraction(g) - Fraction(e, 2 ** TOP)) <= Fraction(5, 2)
        if a == 0.0:
            assert cmul(X, Y, w, conj) == [X, Y]


def test_product_by_sqrt_half():
    C = 3260954456333195553
    assert C == round(Fraction(math.isqrt(2 ** 199), 2 ** 100) * 2 ** TOP)
    ch, cl = limbs(C)
    rng = random.Random(3)
    for _ in range(2000):
        X = rng.randrange(-2 ** 62 - 2 ** 61, 2 ** 62 + 2 ** 61)   # a sum of two components
        xh, xl = limbs(X)
        got = chk(chk(4 * chk(xh * ch)) + (chk((1 << 29) + xh * cl + xl * ch) >> 30))
        assert abs(got - Fraction(X * C, 2 ** TOP)) <= Fraction(3, 2)


def fx_in(v, sh):
    """fx_in: the mantissa at the top of a word, down by 1085 - sh - e, one more bit rounding."""
    m, e = math.frexp(abs(v))
    t = 1085 - sh - (e + 1022)
    top = int(m * 2 ** 53) << 11 if v else 0
    q = ((top >> t if t < 64 else 0) + 1) >> 1
    return -q if v < 0 else q


def fx_out(X, sh):
    """fx_out_int: the nearest double, ties to even, by integer operations."""
    a = abs(X)
    if a == 0:
        return 0.0
    m = a << (63 - a.bit_length())
    q = (m + 0x1FF + ((m >> 10) & 1)) >> 10
    field = a.bit_length() + 1021 - sh + (q >> 52)
    return math.copysign(math.ldexp(1.0 + (q & (2 ** 52 - 1)) / 2.0 ** 52, field - 1023), X)


@pytest.mark.parametrize("G", [2, 9, 13, 15])
def test_conversions(G):
    rng = random.Random(G)
    sh = TOP - G        # a line whose largest value is just below 1
    for _ in range(4000):
        v = rng.uniform(-1, 1) * 2.0 ** -rng.choice([0, 0, 1, 5, 40, 60, 70])
        x = fx_in(v, sh)
        assert abs(x - Fraction(v) * 2 ** sh) <= Fraction(1, 2)
        assert abs(x) <= 2 ** (TOP - G)
        y = rng.randrange(-2 ** rng.randint(1, 62), 2 ** 62)
        assert fx_out(y, sh) == float(Fraction(y, 2 ** sh))
    for y in (2 ** 53 + 1, 2 ** 53 + 3, 2 ** 62 - 1, 2 ** 54 - 1, 1, -1, 0):
        assert fx_out(y, sh) == float(Fraction(y, 2 ** sh))
