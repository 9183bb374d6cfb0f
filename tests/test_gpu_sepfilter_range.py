"""The separable filters (csrc/sepfilter.cu) of fields whose values one scale per CTA
does not cover: a jet over a field 1e9 times weaker, and values and weights at
the ends of the exponents.  The face-filtered velocity,
which no projection spreads, against the oracle: a filtered value is three nested
sums of at most 17 products with weights of one sign, 51 2^-53 = 5.7e-15 of the
sum of magnitudes; 1e-14 relative L2 in every part of the field."""
import numpy as np
import pytest

from oracle import ns

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def NS(built_lib):
    from exactclosure_gb300 import navierstokes

    return navierstokes


def face_filtered(NS, u, c, fdelta):
    d = NS.DnsAid(u.shape[1], 1.0, 1e-3, c, fdelta)
    d.set_velocity(u)
    d.set_paper(True, "surface")
    d.start()
    out = d.get("fu")
    d.close()
    return out


@pytest.mark.parametrize("axis", [1, 2, 3])
def test_jet_over_a_weak_field(NS, axis):
    n, c = 100, 5
    f = ns.gaussian(1 / n, 2 * c / n, 2)
    x = np.arange(n)
    jet = np.exp(-(((x - 25) / 4.0) ** 2)).reshape([n if a == axis else 1 for a in range(1, 4)])
    # one sign: no cancellation in the sums
    u = jet[None] + 1e-9 * np.random.default_rng(axis).uniform(0.5, 1.5, (3, n, n, n))
    got, ref = face_filtered(NS, u, c, f), ns.face_filter(u, c, f)
    for part in (slice(0, 10), slice(11, 19)):
        i = tuple([slice(None)] + [part if a == axis else slice(None) for a in range(1, 4)])
        assert np.linalg.norm(got[i] - ref[i]) < 1e-14 * np.linalg.norm(ref[i])


@pytest.mark.parametrize("field,weight", [(-790, -190), (-420, -190), (0, -190), (-790, -60), (700, 100), (-960, 0)])
def test_small_and_large_exponents(NS, field, weight):
    n, c = 50, 5
    f = ns.gaussian(1 / n, 2 * c / n, 2)
    u = np.random.default_rng(1).uniform(0.5, 1.5, (3, n, n, n))
    got = face_filtered(NS, np.ldexp(u, field), c, np.ldexp(f, weight))  # the Gaussian enters once per axis
    ref, e = ns.face_filter(u, c, f), field + 3 * weight
    if e < -1100:  # below the smallest double
        assert (got == 0).all()
    else:
        assert np.linalg.norm(np.ldexp(got, -e) - ref) < 1e-14 * np.linalg.norm(ref)
