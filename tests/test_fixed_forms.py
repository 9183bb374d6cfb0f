"""CPU checks of the fixed-point arithmetic of csrc/fixed.cuh and its users,
restated in Python integers:

* the FP64 sweep (csrc/rhs.cu): velocities as integers of 57 bits below a power of
  two, split in halves of 29 bits; stress and divergence in three sums, 2 visc/h
  outside them where it is far from the velocities.  Every partial sum stays
  below 2^63, every half in 32 bits, and a component's error against exact
  rationals is no larger than that of the FP64 arithmetic
  (test_fp64_forms.shifted_rhs) down to 2^-4 of the scale, where the sweep
  leaves a weak component to FP64;
* the Burgers filters (csrc/burgers.cu): sums of 511 taps stay below 2^63, of 3001
  they do not;
* the box sums (csrc/filter.cu): K values rounded to 58 bits below the largest, off by at
  most K 2^-58 of it and half a unit of the sum.
"""
import math
from fractions import Fraction

import numpy as np
import pytest

from test_fp64_forms import shifted_rhs

AX = {0: 2, 1: 1, 2: 0}  # axes of u[c]: z, y, x


def at(a, d, s):
    return np.roll(a, -s, axis=AX[d])


def halves(U, low):
    h = (U + (1 << (low - 1))) >> low
    return h, U - (h << low)


class Sum:
    """Three sums of products of halves, checked against int64."""

    def __init__(self, low):
        self.low, self.s, self.most = low, [0, 0, 0], 0

    def mac(self, a, b):
        (ah, al), (bh, bl) = halves(a, self.low), halves(b, self.low)
        for v in (ah, al, bh, bl):
            assert max(abs(v.min()), abs(v.max())) < 2**31
        for i, p in enumerate((ah * bh, ah * bl, al * bh, al * bl)):
            k = (0, 1, 1, 2)[i]
            self.s[k] = self.s[k] + p
            self.most = max(self.most, abs(self.s[k].min()), abs(self.s[k].max()))

    def value(self):
        assert self.most < 2**63
        return (self.s[0] << 2 * self.low) + (self.s[1] << self.low) + self.s[2]


def exponent(x):
    return math.frexp(x)[1]


def to_int(u, e, bits):
    return np.frompyfunc(lambda v: round(Fraction(float(v)) * Fraction(2) ** (bits - e)), 1, 1)(u)


def sweep(u, visc, h, bits=57, low=29):
    """du of the fixed-point sweep with the scale of the whole grid, as rationals."""
    S, m = 2 * visc / h, np.abs(u).max()
    E = exponent(m)
    apart = abs(S) > 2.0 ** (E - 1) or abs(S) < 2.0 ** (E - 6)  # S outside the integers
    if not apart:
        E = exponent(max(m + abs(S), 4 * abs(S)))
    U = to_int(u, E, bits)
    S4 = 0 if apart else (round(Fraction(4 * S) * Fraction(2) ** (bits - E)) + 2) >> 2 << 2
    S2 = S4 >> 1
    full = lambda v: v + 0 * U[0]
    out = []
    for i in range(3):
        s, a = Sum(low), U[i]
        d = at(a, i, 1) - at(a, i, -1)
        s.mac(d, at(a, i, 1) + at(a, i, -1) + 2 * a - S4)
        linear = -4 * d
        group = 0
        for j in range(3):
            group = group + (a - at(a, j, -1)) + (U[j] - at(U[j], j, -1))
            if j == i:
                continue
            A, B = a + at(a, j, 1) - S2, U[j] + at(U[j], i, 1) - S2
            s.mac(A, B)
            s.mac(-at(A, j, -1), at(B, j, -1))
            linear = linear - 2 * (A + B - at(A + B, j, -1))
            if not apart:
                s.mac((a - at(a, j, -1)) + (U[j] - at(U[j], j, -1)), full(S4))
        if not apart:
            s.mac(2 * (a - at(a, i, -1)), full(S4))
        linear = linear + 4 * group
        unit = Fraction(2) ** (E - bits)
        r = np.frompyfunc(lambda v, l: -(v * unit * unit + (Fraction(S) * unit * l if apart else 0)) / (4 * Fraction(h)), 2, 1)
        out.append(r(s.value(), linear))
    return np.array(out)


def exact(u, visc, h):
    f = np.frompyfunc(lambda v: Fraction(float(v)), 1, 1)(u)
    h, rv = Fraction(h), 4 * Fraction(visc) / Fraction(h)
    sig = {}
    for i in range(3):
        a, b = f[i], at(f[i], i, -1)
        sig[i, i] = (a + b) * (a + b) - 2 * rv * (a - b)
        for j in range(i + 1, 3):
            a, b, c, d = f[i], at(f[i], j, 1), f[j], at(f[j], i, 1)
            sig[i, j] = sig[j, i] = (a + b) * (c + d) - rv * ((b - a) + (d - c))
    return np.array([-sum((at(sig[i, i], i, 1) - sig[i, i]) if i == j else (sig[i, j] - at(sig[i, j], j, -1))
                          for j in range(3)) / (4 * h) for i in range(3)])


def error(a, ref):
    """Relative L2 error of each component; exact differences."""
    def norm(x):
        return math.sqrt(float(sum(v * v for v in x.ravel())))
    to = np.frompyfunc(lambda v: v if isinstance(v, Fraction) else Fraction(float(v)), 1, 1)
    return [norm(to(a[i]) - ref[i]) / norm(ref[i]) if norm(ref[i]) else norm(to(a[i])) for i in range(3)]


@pytest.mark.parametrize("visc", [0.0, 1e-30, 1e-5, 1 / 2000, 0.1, 10.0, -0.02])
@pytest.mark.parametrize("k", [0, 2, 3])
def test_sweep_is_no_less_exact_than_fp64(visc, k):
    n = 6
    h = 1.0 / n
    u = np.random.default_rng(k).standard_normal((3, n, n, n))
    u[2] *= 2.0**-k
    ref = exact(u, visc, h)
    for f, e in zip(error(sweep(u, visc, h), ref), error(shifted_rhs(u, visc, h), ref)):
        assert f <= e, (f, e)


@pytest.mark.parametrize("visc", [1 / 2000, 1e-5, 1e-12, 1e-30])
def test_sweep_of_a_shear_flow(visc):
    n = 6
    u = np.zeros((3, n, n, n))
    u[0] = np.random.default_rng(5).standard_normal(n)[None, :, None]
    ref = exact(u, visc, 1.0 / n)
    got = error(sweep(u, visc, 1.0 / n), ref)
    # the velocity's own rounding, 2^-58 of the scale, through second differences
    assert got[0] <= 2.0**-53 and got[1:] == [0, 0]


def test_sweep_sums_at_their_largest():
    """Velocities at both ends of the scale, in every alternation of signs."""
    for s in range(8):
        u = np.array([(-1.0) ** (((s >> c) & 1) + np.indices((4, 4, 4)).sum(axis=0) * (c != s % 3)) for c in range(3)])
        u *= 1 - 2.0**-40
        for visc in (0.0, 0.06, -0.06, 0.002, 1.0):
            sweep(u, visc, 0.25)


@pytest.mark.parametrize("taps,fits", [(511, True), (3001, False)])
def test_burgers_sums(taps, fits):
    x = np.full(taps, to_int(np.array([1.99]), 1, 54)[0], dtype=object)
    w = 1.0 / taps
    s = Sum(27)
    for a, b in zip(to_int(np.full(taps, w), exponent(w), 54), x):
        s.mac(np.array([a], dtype=object), np.array([b], dtype=object))
    assert (s.most < 2**63) == fits


def sum_fixed(v, up=5):
    e = max(math.frexp(x)[1] for x in v)
    t = sum(int(math.copysign((math.floor(Fraction(abs(x)) * Fraction(2) ** (53 + up + 1 - e)) + 1) >> 1, x)) for x in v)
    assert abs(t) < 2**63
    return float(Fraction(t) * Fraction(2) ** (e - 53 - up))


@pytest.mark.parametrize("K", [9, 16, 25])
def test_box_sums(K):
    r = np.random.default_rng(K)
    for _ in range(200):
        v = [float(x) for x in r.standard_normal(K) * np.exp(4 * r.standard_normal(K))]
        ref = sum(Fraction(x) for x in v)
        big = max(map(abs, v))
        assert abs(Fraction(sum_fixed(v)) - ref) <= Fraction(K * big) / 2**58 + abs(ref) / 2**53
