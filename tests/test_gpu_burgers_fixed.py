"""The Burgers DNS-aided LES loop's fixed-point filters and register-resident
velocity (csrc/burgers.cu) where they can go wrong: grid sizes at the edges of
the cells-per-thread variants, a sample that ends inside a thread's cells, long
and short stencils, magnitudes far from one and a mean flow.  Three Euler steps
against the oracle at 1e-12 of each field's largest value: a filtered value
rounds its inputs to 2^-55 of the largest |u| (or of the stress bound, at most
eight times the largest stress) and once more, a few hundred 2^-53 over three
steps of order-one operations."""
import numpy as np
import pytest

from oracle import burgers as ob

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def GB(built_lib):
    from exactclosure_gb300 import burgers

    return burgers


def start(nh, ns, seed, scale, mean):
    r = np.random.default_rng(seed)
    k = np.arange(nh // 2 + 1)
    amp = (k / 3) ** 4 * np.exp(-2 * (k / 3) ** 2)
    a = np.fft.irfft(amp * np.exp(2j * np.pi * r.random((ns, nh // 2 + 1))) * nh, nh, axis=1)
    return scale * (a / np.abs(a).max() + mean)


@pytest.mark.parametrize("nh,nH,delta,kind,scale,mean", [
    (75, 15, 2.0, "gaussian", 1.0, 0.0), (2535, 169, 1.0, "tophat", 1.0, 0.0), (2565, 171, 2.0, "gaussian", 1.0, 0.0),
    (5635, 161, 3.0, "gaussian", 1.0, 0.0), (8775, 325, 2.0, "tophat", 1.0, 0.0), (11775, 785, 2.0, "gaussian", 1.0, 0.0),
    (13815, 921, 2.0, "gaussian", 1.0, 0.0), (13839, 659, 1.0, "gaussian", 1.0, 0.0),
    (2565, 171, 2.0, "gaussian", 1e-6, 0.0), (2565, 171, 2.0, "gaussian", 1e6, 0.0), (2565, 171, 2.0, "gaussian", 1.0, 50.0)])
def test_three_steps(GB, nh, nH, delta, kind, scale, mean):
    L, visc, ns = 2 * np.pi, 5e-4 * scale, 3
    u0 = start(nh, ns, nh, scale, mean)
    b = GB.Batch(GB.Grid(L, nh), ns, visc)
    b.set_velocity(u0)
    b.les_setup(GB.Grid(L, nH), delta, kind)
    tstop = 10.0 / scale  # far beyond three steps
    b.advance(tstop, 0.3, "euler", max_steps=3)
    u, t, steps, V = ob.dns_aided_les(u0, nH, visc, L, delta, kind, tstop, 0.3, max_steps=3)
    assert np.abs(b.velocity() - u).max() <= 1e-12 * np.abs(u).max()
    assert np.abs(b.time()[0] - t).max() <= 1e-13 * t.max() and (b.time()[1] == steps).all()
    for k in ob.LES_NAMES:
        assert np.abs(b.les(k) - V[k]).max() <= 1e-12 * np.abs(V[k]).max(), k
    b.close()


def test_zero_field_stays_zero(GB):
    b = GB.Batch(GB.Grid(2 * np.pi, 225), 2, 5e-4)
    b.set_velocity(np.zeros((2, 225)))
    b.les_setup(GB.Grid(2 * np.pi, 45), 2.0, "gaussian")
    b.advance(1.0, 0.3, "euler", max_steps=2)
    for k in ob.LES_NAMES:
        assert (b.les(k) == 0).all()
    b.close()
