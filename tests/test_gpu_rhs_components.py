"""The FP64 sweep (csrc/rhs.cu) component by component, where its one scale for the
three of them could cost a weak one its digits.

Tolerance of component i, with m_i its largest value, M the largest of all and
r = 4 visc/h: the FP64 arithmetic sums six stress terms of up to 4 m_i M + 4 r M
with about five roundings each over 4h, 30 2^-53 (m_i M + r M)/h.  The
fixed-point path rounds its inputs to 2^-58 of at most 4 M, through six
products of two-point sums (48 2^-58 M M/h), and is taken for m_i >= 2^-5 M, so
that is at most 48 2^-53 m_i M/h.  Twice their sum."""
import numpy as np
import pytest

from test_gpu_rhs_fixed import exact_rhs, run

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def NS(built_lib):
    from exactclosure_gb300 import navierstokes

    return navierstokes


def limits(u, visc):
    n = u.shape[1]
    m = np.abs(u).max(axis=(1, 2, 3))
    return 2 * 78 * 2.0**-53 * (m * m.max() + 4 * abs(visc) * n * m.max()) * n


def check(NS, u, visc):
    got, ref = run(NS, u, visc), exact_rhs(u, visc)
    err = np.abs(got - ref).max(axis=(1, 2, 3))
    assert (err <= limits(u, visc)).all(), (err, limits(u, visc))


@pytest.mark.parametrize("visc", [1 / 2000, 1e-5, 1e-30])
@pytest.mark.parametrize("k", [3, 4, 5, 6, 7, 8, 12, 30, 60])
def test_weak_component(NS, k, visc):
    for c, n in ((0, 16), (1, 40), (2, 70)):
        u = np.random.default_rng(k).standard_normal((3, n, n, n))
        u[c] *= 2.0**-k
        check(NS, u, visc)


def test_weak_in_part_of_the_grid(NS):
    """A component that is weak in some tiles and planes only."""
    n = 66
    u = np.random.default_rng(1).standard_normal((3, n, n, n))
    u[2, 20:50] *= 1e-9
    u[1, :, 16:48, :] *= 1e-7
    check(NS, u, 1e-30)


def test_component_of_zeros(NS):
    """Beside strong ones: only the viscous term reaches it."""
    n = 66
    u = np.random.default_rng(1).standard_normal((3, n, n, n))
    u[2, 20:50] *= 1e-9
    u[1, :, 16:48, :] *= 1e-7
    u[0] = 0
    check(NS, u, 1e-30)


@pytest.mark.parametrize("kind", ["noise", "wave"])
@pytest.mark.parametrize("visc", [1 / 500, 1 / 2000, 1e-5, 1e-7, 1e-12, 1e-30])
def test_shear_flow(NS, visc, kind):
    """u_1(y) alone: the advection terms cancel exactly and the viscous ones are
    left, 30 2^-53 r M / h in FP64 and 24 2^-58 4 M r / 4 / h in fixed point."""
    for n in (16, 66):
        f = np.random.default_rng(n).standard_normal(n) if kind == "noise" else np.sin(2 * np.pi * (np.arange(n) + 0.3) / n)
        u = np.zeros((3, n, n, n))
        u[0] = f[None, :, None]
        err = np.abs(run(NS, u, visc) - exact_rhs(u, visc)).max(axis=(1, 2, 3))
        assert (err <= 2 * 31 * 2.0**-53 * 4 * visc * n * np.abs(f).max() * n * np.array([1, 0, 0])).all(), err


@pytest.mark.parametrize("visc", [-1e-4, -1 / 50, -0.1])
def test_negative_viscosity(NS, visc):
    """What a time reversal passes; r is its magnitude."""
    for n in (16, 66):
        check(NS, np.random.default_rng(n).standard_normal((3, n, n, n)), visc)


@pytest.mark.parametrize("scale", [1.0, 1e-20])
@pytest.mark.parametrize("visc", [1 / 500, 0.02, 0.1, 10.0, -10.0, 1e6])
def test_viscosity_beside_a_weak_velocity(NS, visc, scale):
    """2 visc/h about the velocity and far above it."""
    for n in (16, 40, 66):
        u = np.random.default_rng(n).standard_normal((3, n, n, n)) * scale
        u[:, n // 2:] *= 0.01
        check(NS, u, visc)


def test_still_planes(NS):
    """Zeros beside a moving half: no scale of their own."""
    for n in (16, 66):
        u = np.random.default_rng(n).standard_normal((3, n, n, n))
        u[:, 2: n - 3] = 0
        check(NS, u, 1 / 500)
        assert (run(NS, u, 1 / 500)[:, 3: n - 4] == 0).all()
