"""The quotient of the gate/up epilogue (csrc/quotient.cuh, div8) restated with exactly rounded single-precision steps."""
from fractions import Fraction

import numpy as np

F, BITS = np.float32, 23
LEFT_OUT = range((1 << BITS) - 5, 1 << BITS)             # mantissas that take the division itself


def _fma(a, b, c):
    """a b + c rounded once: the product is exact in the 64 bits of an x87 mantissa, the sum is rounded to odd there, then to single."""
    p, c = a.astype(np.longdouble) * b.astype(np.longdouble), c.astype(np.longdouble)
    s = p + c
    t = s - p
    e = (p - (s - t)) + (c - t)                       # what the sum dropped
    m = s.view(np.uint64)[::2]                        # its mantissa
    inexact, up = e != 0, (e < 0) == (s > 0)
    m[...] = np.where(inexact & up & (m & 1 == 0) & (m != 1 << 63), m - 1, np.where(inexact & ~up, m | 1, m))
    return s.astype(F)


def _quotient(a, d, y):
    q = a * y
    return _fma(_fma(-q, d, a), y, q)


def _mantissas(n=1 << BITS):
    return (np.arange(n, dtype=np.int32) + (127 << BITS)).view(F)


def _near_ties(m, width=64):
    """Dividends in [1, 2) whose quotient by 1 + m / 2^23 lies within width 2^-48 of half-way between two floats, to either side of it
    or on a float: a reciprocal that is off by units of the last place moves the corrected quotient by less, and only they can turn."""
    D = (1 << BITS) + m
    out = set()
    for shift in (24, 25):                            # quotients from 1 on, and below: a 2^shift = (2 k + 1) D + r or 2 k D + r
        for r in range(-width, width + 1):
            for odd in (0, 1):
                # x D = -r modulo 2^shift for the quotient's last bits x, x odd or even
                z = (D & -D).bit_length() - 1
                if r % (1 << z):
                    continue
                mod = 1 << (shift - z)
                x0 = (-r >> z) * pow(D >> z, -1, mod) % mod
                for x in range(x0, 1 << 25, mod):
                    A, rest = divmod(x * D + r, 1 << shift)
                    if rest == 0 and x % 2 == odd and 1 << BITS <= A < 1 << (BITS + 1):
                        out.add(A - (1 << BITS))
    return sorted(out)


def test_where_one_newton_step_is_not_enough():
    """From every estimate within two units of the last place (the instruction's bound is a relative 2^-23)."""
    d = _mantissas()
    right = (np.longdouble(1) / d.astype(np.longdouble)).astype(F)
    wrong, spoilt = set(), set()
    for off in (-2, -1, 0, 1, 2):
        y = (right.view(np.int32) + off).view(F)
        y = _fma(_fma(-d, y, np.ones_like(d)), y, y)
        wrong |= {(int(i), y[i]) for i in np.nonzero(y != right)[0]}
    assert len(wrong) > 30 and all(abs(int(np.float32(y).view(np.int32)) - int(right[i].view(np.int32))) == 1 for i, y in wrong)
    for i, y in wrong:
        a = d[_near_ties(i)]
        dd = np.full_like(a, d[i])
        bad = _quotient(a, dd, np.full_like(a, y)) != a / dd
        spoilt |= {i} if bad.any() else set()
    assert spoilt and spoilt <= set(LEFT_OUT), spoilt


def test_corrected_quotient_is_the_division():
    """With the right reciprocal: dividends and divisors at random, and every dividend near a tie of divisors at random."""
    rng, d = np.random.default_rng(0), _mantissas()
    y = (np.longdouble(1) / d.astype(np.longdouble)).astype(F)
    a = d[rng.permutation(d.size)]
    assert np.array_equal(_quotient(a, d, y), a / d)
    for m in rng.integers(0, 1 << BITS, 100).tolist() + [0, 1, 2, (1 << BITS) - 6]:
        a = d[_near_ties(m)]
        q = a / d[m]
        assert np.array_equal(_quotient(a, np.full_like(a, d[m]), np.full_like(a, y[m])), q)
        for x, z in zip(a[:3], q[:3]):                # (the oracle itself, in rational numbers)
            exact = Fraction(float(x)) / Fraction(float(d[m]))
            assert all(abs(exact - Fraction(float(z))) <= abs(exact - Fraction(float(np.nextafter(z, F(t))))) for t in (0, 4))
