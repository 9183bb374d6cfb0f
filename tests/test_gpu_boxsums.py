"""Transverse box sums with the ratio compiled in (FP64 on the integer pipe)
against NumPy: magnitudes spread over many orders, signs, zeros, tiny and
non-finite values, ratios with and without a kernel of their own.  A value is a
mean of c^2 numbers, each taken to 2^-57 of the block's largest and the sum
rounded once: 2^-51 of the block's largest magnitude bounds the error of the two
passes; FP32 sums of up to 64 terms: 2^-20."""
import numpy as np
import pytest

from oracle import ns

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n,c", [(24, 2), (24, 3), (32, 4), (20, 5), (36, 6), (48, 8)])
@pytest.mark.parametrize("spread,scale", [(0, 0), (12, 0), (30, 0), (3, -930), (3, 960)])
def test_face_targets(built_lib, n, c, precision, spread, scale):
    from exactclosure_gb300 import navierstokes as NS

    if precision == 1 and (scale or spread > 12):
        scale, spread = 0, 12
    rng = np.random.default_rng(n + spread)
    u = rng.normal(size=(3, n, n, n)) * 2.0 ** rng.uniform(-spread, spread, size=(3, n, n, n))
    u[:, 1, 2, :] = 0.0
    u = np.ldexp(u, scale)
    if precision == 1:
        u = u.astype(np.float32).astype(np.float64)
    cs = NS.Case(n, 1.0, 1e-3, 0.3, precision=precision, les=[(c, "face")])
    cs.set_velocity(u)
    got = np.ldexp(cs.les(0, "target"), -scale)
    ref = ns.filtered_target(np.ldexp(u, -scale), ns.Les(c=c, kind="face"), 1.0)
    size = ns.filtered_target(np.abs(np.ldexp(u, -scale)), ns.Les(c=c, kind="face"), 1.0)
    tol = 2.0**-51 if precision == 0 else 2.0**-20
    assert (np.abs(got - ref) <= tol * c * c * size).all()
    cs.close()


@pytest.mark.parametrize("c", [2, 3, 4, 5])
def test_a_non_finite_cell_stays_in_its_blocks(built_lib, c):
    from exactclosure_gb300 import navierstokes as NS

    n = 12 * c if c == 5 else 24
    u = np.random.default_rng(c).normal(size=(3, n, n, n))
    cs = NS.Case(n, 1.0, 1e-3, 0.3, les=[(c, "face")])
    cs.set_velocity(u)
    ref = cs.les(0, "target")
    u[0, 0, 1, c - 1] = np.inf
    cs.set_velocity(u)
    got = cs.les(0, "target")
    bad = ~np.isfinite(got)
    assert bad.sum() == 1 and np.isposinf(got[bad]).all()
    assert (got[~bad] == ref[~bad]).all()
    cs.close()
