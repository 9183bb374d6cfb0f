"""The batched coarse-grid work of a stage (csrc/lesstep.cu) where it can go
wrong: the smallest LES grids, odd ratios and both filters, rows that are no
multiple of a block, the first LES grid of the mixed-precision solve (one slot
at a time), several LES, and the learned state's slot.  Tolerances are those
of the stepper against the oracle: 1e-12 relative L2 in FP64; 2e-5 in FP32
(states of order one after two steps, 1e-7 a rounding)."""
import numpy as np
import pytest

from oracle import ns

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def NS(built_lib):
    from exactclosure_gb300 import navierstokes

    return navierstokes


def rel(a, b):
    return float(np.linalg.norm((a - b).ravel()) / np.linalg.norm(b.ravel()))


@pytest.mark.parametrize("precision,tol", [(0, 1e-12), (1, 2e-5)])
@pytest.mark.parametrize("n,les", [(8, [(2, "volume"), (2, "face")]), (20, [(5, "face")]), (36, [(2, "volume"), (3, "volume")]),
                                   (68, [(2, "volume")]), (168, [(2, "volume")])])
def test_states_targets_and_pairs(NS, n, les, precision, tol):
    l, visc, cfl = 1.0, 1 / 500, 0.3
    u = ns.randomfield(n, l, 3, 5)
    cs = NS.Case(n, l, visc, cfl, precision=precision, les=les)
    cs.set_velocity(u)
    ol = [ns.Les(c=c, kind=k) for c, k in les]
    steps = 1 if n > 100 else 2
    u, _, closures = ns.dnsaid_rk4(u, visc, l, cfl, steps, ol, record_closure=True)
    cs.step(steps)
    assert rel(cs.velocity(), u) < tol
    for i, le in enumerate(ol):
        assert rel(cs.les(i, "exact"), le.v_exact) < tol
        assert rel(cs.les(i, "nomodel"), le.v_nomodel) < tol
        assert rel(cs.les(i, "target"), ns.filtered_target(u, le, l)) < tol
        # stage 0 of the last step; the closure is a difference of terms the
        # size of the right-hand side
        _, ub, m = closures[(steps - 1) * len(ol) + i]
        assert rel(cs.les(i, "target_last"), ub) < tol
        size = np.linalg.norm(ns.rhs(ub, visc, l * le.c / n))
        assert np.linalg.norm(cs.les(i, "closure") - m) < tol * size
    cs.close()
