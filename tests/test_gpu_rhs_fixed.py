"""The FP64 right-hand side's fixed-point sweep (csrc/rhs.cu) against extended
precision at the sizes and values where it can go wrong: grids smaller than a
tile and at its edges, fields that are not 16-byte aligned, magnitudes that
change by many binades from plane to plane (the shared exponent moves) or
inside a tile (cells that take the FP64 arithmetic), values out of the
fixed-point range, zeros, infinities and NaN.

Tolerance: per cell, with m the largest |u| of the 3^3 cells around it, the
FP64 arithmetic the sweep replaces sums six stress terms of up to 4 m^2 + 4 r m
(r = 4 visc/h) with about five roundings each, over 4h: 30 2^-53 (m^2 + r m)/h.
The fixed-point path adds its conversion, 2^-58 of at most 4 (2^7 m + r) per
value, through six products of two-point sums: 12 m 2^-49 m / h, another 192
2^-53 of the same.  Twice their sum bounds both paths."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
LD = np.longdouble


@pytest.fixture(scope="module")
def NS(built_lib):
    from exactclosure_gb300 import navierstokes

    return navierstokes


def at(a, d, s):
    return np.roll(a, -s, axis=(2, 1, 0)[d]) if s else a


def exact_rhs(u, visc):
    n = u.shape[1]
    h, u, visc = LD(1) / n, u.astype(LD), LD(visc)
    s = {}
    for i, j in ((0, 0), (1, 1), (2, 2), (0, 1), (1, 2), (2, 0)):
        o = int(i != j)
        a, b, c, d = at(u[i], j, o), at(u[i], j, o - 1), at(u[j], i, o), at(u[j], i, o - 1)
        s[i, j] = s[j, i] = (a + b) * (c + d) / 4 - visc * ((a - b) + (c - d)) / h
    out = np.zeros_like(u)
    for i in range(3):
        for j in range(3):
            out[i] -= ((at(s[i, j], j, 1) - s[i, j]) if i == j else (s[i, j] - at(s[i, j], j, -1))) / h
    return out


def bound(u, visc):
    n = u.shape[1]
    m = np.abs(u).max(axis=0)
    for d in range(3):
        m = np.maximum(m, np.maximum(at(m, d, 1), at(m, d, -1)))
    r = 4 * visc * n
    return 2 * 222 * 2.0**-53 * (m * m + r * m + r * r * 2.0**-5) * n


def field(kind, n):
    r = np.random.default_rng(n)
    u = r.standard_normal((3, n, n, n))
    if kind == "planes":  # 24 decades over z, up and down
        u *= (10.0 ** (-12 * np.cos(2 * np.pi * np.arange(n) / n)))[None, :, None, None]
    elif kind == "jet":
        x = 2 * np.pi * np.arange(n) / n
        d = sum((q - 3.0) ** 2 for q in np.meshgrid(x, x, x, indexing="ij"))
        u = np.exp(-8 * d)[None] * np.array([1.0, 0.5, -0.2])[:, None, None, None] + 1e-9 * u
    elif kind == "rest":  # zero but for one corner
        u[:, n // 2:] = 0
    elif kind == "large":
        u *= 1e30
    elif kind == "small":
        u *= 1e-60
    return u


def run(NS, u, visc, doadd=False, unaligned=False):
    import torch

    n = u.shape[1]
    buf = torch.empty(u.size + 1, dtype=torch.float64, device="cuda")
    t = buf[1:] if unaligned else buf[:-1]
    t = t.view(3, n, n, n).copy_(torch.from_numpy(u))
    out = torch.ones_like(t)
    NS.tensordivergence(out, t, visc, NS.Grid(1.0, n), doadd)
    return out.cpu().numpy()


@pytest.mark.parametrize("n", [4, 6, 16, 18, 30, 32, 34, 36, 50, 66, 100])
def test_grid_sizes(NS, n):
    u = field("noise", n)
    got = run(NS, u, 1 / 2000)
    ref = exact_rhs(u, 1 / 2000)
    assert (np.abs(got - ref) <= bound(u, 1 / 2000)).all()
    # the result is rounded twice: no worse than the FP64 arithmetic overall
    assert np.sqrt(((got - ref) ** 2).sum() / (ref**2).sum()) < 2e-16


@pytest.mark.parametrize("kind", ["planes", "jet", "rest", "large"])
@pytest.mark.parametrize("n", [40, 66])
def test_magnitudes(NS, kind, n):
    u = field(kind, n)
    got, ref = run(NS, u, 1 / 2000), exact_rhs(u, 1 / 2000)
    assert (np.abs(got - ref) <= bound(u, 1 / 2000)).all()
    if kind == "rest":
        assert (got[:, n // 2 + 1:n - 1] == 0).all()


@pytest.mark.parametrize("visc", [0.1, 10.0, 1e-30])
def test_viscosities(NS, visc):
    u = field("noise", 40)
    got, ref = run(NS, u, visc), exact_rhs(u, visc)
    assert (np.abs(got - ref) <= bound(u, visc)).all()


def test_small_values(NS):
    u = field("small", 34)
    got, ref = run(NS, u, 1e-62), exact_rhs(u, 1e-62)
    assert (np.abs(got - ref) <= bound(u, 1e-62)).all()


def test_zero_field(NS):
    assert (run(NS, np.zeros((3, 34, 34, 34)), 1 / 2000) == 0).all()


@pytest.mark.parametrize("n", [36, 70])
def test_unaligned_field_and_doadd(NS, n):
    u = field("noise", n)
    a = run(NS, u, 1 / 2000)
    assert (run(NS, u, 1 / 2000, unaligned=True) == a).all()
    assert (run(NS, u, 1 / 2000, doadd=True) == 1 + a).all()


def test_nonfinite_values_stay_where_they_reach(NS):
    u = field("noise", 66)
    u[1, 3, 4, 5] = np.inf
    u[0, 40, 20, 64] = np.nan
    got = run(NS, u, 1 / 2000)
    with np.errstate(all="ignore"):
        ref = exact_rhs(u, 1 / 2000)
        ok = np.isfinite(ref)
        assert (np.isfinite(got) == ok).all()
        v = np.where(np.isfinite(u), u, 10.0)
        assert (np.abs(got - ref) <= bound(v, 1 / 2000))[ok].all()
