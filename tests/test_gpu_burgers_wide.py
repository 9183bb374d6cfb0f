"""Burgers DNS-aided LES with stencils about and beyond the longest that the
fixed-point filters hold (csrc/burgers.cu): top hats, whose equal weights add
coherently, over a nearly uniform velocity just below a power of two, where the
integer sums are largest.  Two Euler steps against the oracle at 1e-12 of each
field's largest value: a sum of T = 3375 FP64 products of weights that add to
one is off by at most T 2^-53 = 4e-13 of it."""
import numpy as np
import pytest

from oracle import burgers as ob

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def GB(built_lib):
    from exactclosure_gb300 import burgers

    return burgers


@pytest.mark.parametrize("nh,nH,delta,taps", [(1500, 300, 101.4, 511), (1500, 300, 101.8, 513), (4500, 12, 8.0, 3375)])
def test_wide_top_hats_over_a_mean_flow(GB, nh, nH, delta, taps):
    L, visc, ns = 2 * np.pi, 5e-4, 2
    assert len(GB.filter_kernels(GB.Grid(L, nh), GB.Grid(L, nH), delta, "tophat")[1][1]) == taps
    u0 = 1.99 + 0.005 * np.random.default_rng(nh).standard_normal((ns, nh)).clip(-1, 1)
    b = GB.Batch(GB.Grid(L, nh), ns, visc)
    b.set_velocity(u0)
    b.les_setup(GB.Grid(L, nH), delta, "tophat")
    b.advance(10.0, 0.3, "euler", max_steps=2)
    u, t, steps, V = ob.dns_aided_les(u0, nH, visc, L, delta, "tophat", 10.0, 0.3, max_steps=2)
    assert np.abs(b.velocity() - u).max() <= 1e-12 * np.abs(u).max()
    assert (b.time()[1] == steps).all()
    for k in ob.LES_NAMES:
        assert np.abs(b.les(k) - V[k]).max() <= 1e-12 * np.abs(V[k]).max(), k
    b.close()
