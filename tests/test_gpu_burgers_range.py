"""Burgers samples at the ends of what the shared scales of the fixed-point filters
cover (csrc/burgers.cu): a pulse over a field a million times weaker, which goes
on in FP64 beside samples that stay, and a viscous flow, whose stress is far
below the bound it is scaled by.  One step of the size of a coarse cell against
extended precision, with the tolerance of test_gpu_burgers_closure.py, the cells
away from the pulse by themselves; and several steps in calls of different
lengths against the oracle."""
import numpy as np
import pytest

from oracle import burgers as ob
from test_gpu_burgers_closure import exact_step

pytestmark = pytest.mark.gpu
nH, comp, L = 25, 57, 2 * np.pi
nh = nH * comp


@pytest.fixture(scope="module")
def GB(built_lib):
    from exactclosure_gb300 import burgers

    return burgers


def pulse(seed):
    x = np.arange(nh)
    r = np.random.default_rng(seed)
    return np.exp(-(((x - 300) / 30) ** 2)) + 1e-6 * (1 + 0.5 * np.repeat(r.uniform(-1, 1, nH), comp))


def wave(seed):
    r = np.random.default_rng(seed)
    return np.repeat(r.uniform(-1, 1, nH), comp) + 0.1 * r.standard_normal(nh)


@pytest.mark.parametrize("visc,start,cells", [(1e-9, pulse, slice(12, 22)), (1.0, wave, slice(None))])
def test_one_step(GB, visc, start, cells):
    u0 = np.stack([start(0), start(1)])
    b = GB.Batch(GB.Grid(L, nh), 2, visc)
    b.set_velocity(u0)
    b.les_setup(GB.Grid(L, nH), 1.0, "gaussian")
    wl, wd = (k[1] for k in GB.filter_kernels(GB.Grid(L, nh), GB.Grid(L, nH), 1.0, "gaussian"))
    V = b.les("nomodel")
    b.advance(1e6, float(comp), "euler", max_steps=1)
    ref = exact_step(u0, V, nH, visc, L, wl, wd, b.time()[0])
    for k in ob.LES_NAMES:
        d, f = (b.les(k) - ref[k])[:, cells], ref[k][:, cells]
        err = float(np.sqrt((d**2).sum() / (f**2).sum()))
        assert err < 8 * 2.0**-53, (k, err)
    b.close()


@pytest.mark.parametrize("visc", [1e-4, 0.02])
def test_samples_that_leave_beside_samples_that_stay(GB, visc):
    u0 = np.stack([wave(3), pulse(4), wave(5) * 0.01, pulse(6), np.zeros(nh)])
    b = GB.Batch(GB.Grid(L, nh), 5, visc)
    b.set_velocity(u0)
    b.les_setup(GB.Grid(L, nH), 2.0, "gaussian")
    state = None
    for steps in (1, 5, 2):
        b.advance(10.0, 0.3, "euler", max_steps=steps)
        state = ob.dns_aided_les(u0, nH, visc, L, 2.0, "gaussian", 10.0, 0.3, max_steps=steps, state=state)
        u, t, n, V = state
        assert (b.time()[1] == n).all() and np.abs(b.time()[0] - t).max() <= 1e-13 * t.max()
        assert np.abs(b.velocity() - u).max() <= 1e-12 * np.abs(u).max()
        for k in ob.LES_NAMES:
            assert np.abs(b.les(k) - V[k]).max() <= 1e-12 * np.abs(V[k]).max(), k
    b.close()
