"""CPU model of the block-fixed-point explicit step's integers (csrc/euler.cu,
bfp_fixed / bfp_scale / bfp_mu), in Python integers against exact rationals:
every 64-bit intermediate in range and mu within its stated error, for fields
from a quench's noise to large values, checkerboards at the top of a binade,
and model constants on either side of the field's scale."""
import math
import random
from fractions import Fraction

import pytest


def chk(v):
    assert -(1 << 63) <= v < (1 << 63), "64-bit overflow"
    return v


def limbs(v):
    lo = ((v + (1 << 31)) & 0xFFFFFFFF) - (1 << 31)
    hi = (v - lo) >> 32
    assert -(1 << 31) <= hi < (1 << 31)
    return hi, lo


def fixed(x, s):
    """bfp_fixed: floor(x 2^(60-s)), one less for whole negative values."""
    X = math.floor(Fraction(abs(x)) * Fraction(2) ** (60 - s))
    return X if math.copysign(1.0, x) > 0 else ~X


def scale(s, c2, eps, dims):
    ls = 2.0 * dims * c2 - eps
    lin = abs(ls) + 2.0 * dims * abs(c2)
    elin = math.frexp(lin)[1] if lin else -4000
    a = max(2 * s, elin)
    lsi = round(Fraction(ls) * Fraction(2) ** (61 - a))
    m, e = math.frexp(abs(c2))
    mc, ec = int(m * 2 ** 53) * 1024 * (1 if c2 >= 0 else -1), e + 1022
    r = a + 1024 - ec
    C = 0 if r > 62 or c2 == 0 else -((mc + (1 << (r - 1))) >> r)
    assert c2 == 0 or r >= 4
    return a, lsi, limbs(chk(C)), ls


def mu(X, S, a, s, lsi, C):
    xh, xl = limbs(X)
    sh, sl = limbs(chk(S))
    G = chk(chk(chk(chk((xh * xh) << 5) + (chk(xh * xl) >> 26)) >> (a - 2 * s)) + lsi)
    assert abs(G) < 1 << 62
    gh, gl = limbs(G)
    mid = chk(sl * C[0])
    for t in (sh * C[1], xl * gh, xh * gl):
        mid = chk(mid + t)
    return chk(chk(xh * gh + sh * C[0]) + (mid >> 32)) >> 1


@pytest.mark.parametrize("dims", [2, 3])
@pytest.mark.parametrize("size", [1e-250, 1e-6, 0.01, 0.99, 40.0, 1e60])
@pytest.mark.parametrize("k,eps", [(1.0, 0.9), (0.0, 0.5), (1e-8, 1e3), (-0.3, 0.9)])
def test_mu_in_integers(dims, size, k, eps):
    rng = random.Random(int(math.log(size) * 7) + dims)
    c2 = 2.0 * k
    s = math.frexp(size)[1]
    a, lsi, C, ls = scale(s, c2, eps, dims)
    unit = Fraction(2) ** (a + s - 56)
    top = math.nextafter(2.0 ** s, 0.0)
    stencils = [[top] * (2 * dims + 1), [top] + [-top] * (2 * dims), [-top] + [top] * (2 * dims), [0.0] * (2 * dims + 1)]
    stencils += [[size * rng.uniform(-1, 1) * 10.0 ** -rng.choice([0, 0, 3, 12]) for _ in range(2 * dims + 1)]
                 for _ in range(150)]
    for v in stencils:
        X = [fixed(x, s) for x in v]
        assert all(abs(x) <= 1 << 60 for x in X)
        M = mu(X[0], sum(X[1:]), a, s, lsi, C)
        assert abs(M) <= (1 << 57) + 4
        # mu of the cut field: M is within the units the kernel's comment states
        p = [x * Fraction(2) ** (s - 60) for x in X]
        want = p[0] * (p[0] * p[0] + Fraction(ls)) - Fraction(c2) * sum(p[1:])
        assert abs(M - want / unit) <= 3
        # and of the field itself, of mu's bound 2^57 units: below 2^-54
        f = [Fraction(x) for x in v]
        want = f[0] * (f[0] * f[0] + Fraction(ls)) - Fraction(c2) * sum(f[1:])
        assert abs(M - want / unit) <= 8
        # the update's exact sum
        assert abs(4 * dims * M) < 1 << 62
