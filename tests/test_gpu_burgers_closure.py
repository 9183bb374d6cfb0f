"""One step of the four Burgers LES (csrc/burgers.cu) against extended precision,
with a time step as large as a coarse cell (the CFL factor is the compression),
so that an error of the filtered quantities shows in the LES states: equal
weights of 1/57 beside the LES kernel [1] or a kernel of their own width.

Tolerance, relative L2: the integer filters round a weight to 2^-54 of its
kernel's largest, a value to 2^-54 of the bound of its quantity and the sum once
(2^-53); the stresses, closures and the update are a dozen FP64 operations on
values of the size of the result.  Independent roundings of a few tenths of
2^-53 each: below 8 2^-53."""
import numpy as np
import pytest

from oracle import burgers as ob

pytestmark = pytest.mark.gpu
LD = np.longdouble


@pytest.fixture(scope="module")
def GB(built_lib):
    from exactclosure_gb300 import burgers

    return burgers


def stress(a, b, visc, h):
    return -((a + b) ** 2) / 8 + visc * (b - a) / h


def exact_step(u, V, nH, visc, L, wl, wd, dt):
    """The states after one forward Euler step of size dt (src/Burgers.jl:397-430)."""
    B, nh = u.shape
    u, V, visc, dt = u.astype(LD), V.astype(LD), LD(visc), dt.astype(LD)[:, None]
    h, H, comp = LD(L) / nh, LD(L) / nH, nh // nH
    s = stress(np.roll(u, 1, 1), u, visc, h)
    face = (np.arange(nH) + 1) * comp - 1
    centre = face - comp // 2

    def filtered(x, w, pos):
        R = len(w) // 2
        return sum(LD(w[r + R]) * x[:, (pos + r) % nh] for r in range(-R, R + 1))

    fsu, vsu, vu = filtered(s, wl, centre), filtered(s, wd, centre), filtered(u, wd, face)
    sVU = stress(filtered(u, wd, centre - 1), filtered(u, wd, centre), visc, h)
    svu = stress(np.roll(vu, 1, 1), vu, visc, H)
    out = {}
    for k, c in zip(ob.LES_NAMES, (0, vsu - sVU, vsu - svu, fsu - svu)):
        q = stress(np.roll(V, 1, 1), V, visc, H) + c
        out[k] = V + dt * (np.roll(q, -1, 1) - q) / H
    return out


@pytest.mark.parametrize("delta", [0.0, 1.0])
def test_one_step_of_the_size_of_a_coarse_cell(GB, delta):
    nH, comp, L, visc = 25, 57, 2 * np.pi, 1e-6
    nh, r = nH * comp, np.random.default_rng(0)
    u0 = np.repeat(r.uniform(-1, 1, (4, nH)), comp, axis=1) + 0.1 * r.standard_normal((4, nh))
    b = GB.Batch(GB.Grid(L, nh), 4, visc)
    b.set_velocity(u0)
    b.les_setup(GB.Grid(L, nH), delta, "tophat")
    wl, wd = (k[1] for k in GB.filter_kernels(GB.Grid(L, nh), GB.Grid(L, nH), delta, "tophat"))
    V = b.les("nomodel")
    b.advance(1e3, float(comp), "euler", max_steps=1)
    ref = exact_step(u0, V, nH, visc, L, wl, wd, b.time()[0])
    for k in ob.LES_NAMES:
        err = float(np.sqrt(((b.les(k) - ref[k]) ** 2).sum() / (ref[k] ** 2).sum()))
        assert err < 8 * 2.0**-53, (k, err)
    b.close()
