"""The separable filters of the LES drivers (csrc/sepfilter.cu) where their
passes can go wrong: a stencil as long as the grid, rows that do not fill the
last CTA, the longest stencil, ratios without a Gaussian and even ones.  Each
driver's first step against the oracle at 1e-12 relative L2: a filtered value
is a weighted mean of at most 40^3 terms, so its FP64 rounding stays below 120
units of 1.1e-16 in three nested sums, the projections and the step add a few
tens more."""
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


@pytest.mark.parametrize("n,c,gauss", [(20, 5, True), (70, 5, True), (66, 3, False), (110, 11, True)])
def test_five_les_step(NS, n, c, gauss):
    l, visc, cfl = 1.0, 1e-3, 0.4
    fdelta = ns.gaussian(l / n, 2 * l * c / n, 2) if gauss else None
    u = ns.randomfield(n, l, -5 / 3, 5, 1.0, profile="power")
    d = NS.DnsAid(n, l, visc, c, fdelta)
    d.set_velocity(u)
    d.start()
    les = ns.dnsaid_start(u, l, c, fdelta)
    d.step(1.0, cfl, max_steps=1)
    u, les, _, _ = ns.dnsaid_project_steps(u, les, visc, l, c, 1.0, cfl, fdelta, max_steps=1)
    assert rel(d.velocity(), u) < 1e-12
    for key in ns.DNSAID_NAMES:
        assert rel(d.get(key), les[key]) < 1e-12, key
    assert rel(d.get("u_les"), ns.apply_DHpi(u, c, l, fdelta)) < 1e-12
    d.close()


@pytest.mark.parametrize("filter,n,c", [("volume", 36, 6), ("surface", 50, 5)])
def test_paper_step_with_gaussian(NS, filter, n, c):
    l, visc, cfl = 1.0, 1e-3, 0.4
    fdelta = ns.gaussian(l / n, 2 * l * c / n, 2)
    u = ns.randomfield(n, l, -5 / 3, 6, 1.0, profile="power")
    d = NS.DnsAid(n, l, visc, c, fdelta)
    d.set_velocity(u)
    d.set_paper(True, filter)
    d.start()
    if filter == "volume":
        steps, fu = ns.dns_aid_volavg_steps, ns.paper_volavg_target(u, l, c, True, fdelta)
    else:
        steps, fu = ns.dns_aid_surface_steps, ns.face_filter(u, c, fdelta)
    assert rel(d.get("fu"), fu) < 1e-12
    les = {k: fu.copy() for k in ns.PAPER_NAMES}
    d.step(1.0, cfl, max_steps=1)
    u, les, _, _ = steps(u, les, visc, l, c, 1.0, cfl, True, fdelta, max_steps=1)
    assert rel(d.velocity(), u) < 1e-12
    for key in ns.PAPER_NAMES:
        assert rel(d.get(key), les[key]) < 1e-12, key
    d.close()


def test_step_of_a_field_with_still_rows(NS):
    """Rows of zeros, which the x pass keeps in FP64, beside moving ones in fixed
    point."""
    n, c, l, visc, cfl = 50, 5, 1.0, 1e-3, 0.4
    fdelta = ns.gaussian(l / n, 2 * l * c / n, 2)
    u = ns.randomfield(n, l, -5 / 3, 5, 1.0, profile="power")
    u[:, n // 2 :] = 0.0
    d = NS.DnsAid(n, l, visc, c, fdelta)
    d.set_velocity(u)
    d.start()
    les = ns.dnsaid_start(u, l, c, fdelta)
    d.step(1.0, cfl, max_steps=1)
    u, les, _, _ = ns.dnsaid_project_steps(u, les, visc, l, c, 1.0, cfl, fdelta, max_steps=1)
    for key in ns.DNSAID_NAMES:
        assert rel(d.get(key), les[key]) < 1e-12, key
    assert rel(d.get("u_les"), ns.apply_DHpi(u, c, l, fdelta)) < 1e-12
    d.close()
