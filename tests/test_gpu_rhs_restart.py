"""The FP64 sweep where its shared exponent moves at every plane (csrc/rhs.cu): the
planes are loaded and converted again while the warps of a CTA still hold the
one before.  Grids whose tiles are TMA boxes (70), 16-byte pieces (34) and words
(an odd first word), against extended precision with the cell-wise bound of
test_gpu_rhs_fixed.py, and equal bits over repeated launches."""
import numpy as np
import pytest

from test_gpu_rhs_fixed import bound, exact_rhs, run

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def NS(built_lib):
    from exactclosure_gb300 import navierstokes

    return navierstokes


@pytest.mark.parametrize("unaligned", [False, True])
@pytest.mark.parametrize("n", [34, 70])
def test_exponent_moves_at_every_plane(NS, n, unaligned):
    u = np.random.default_rng(n).standard_normal((3, n, n, n))
    # by 2, 16 and 2^-5 in turn, and back: up by one binade, up by several, down
    u *= 2.0 ** np.cumsum(np.resize([1, 4, -5], n) * np.where(np.arange(n) % 6 < 3, 1, -1))[None, :, None, None]
    ref, lim = exact_rhs(u, 1 / 2000), bound(u, 1 / 2000)
    first = run(NS, u, 1 / 2000, unaligned=unaligned)
    assert (np.abs(first - ref) <= lim).all()
    for _ in range(20):
        assert (run(NS, u, 1 / 2000, unaligned=unaligned) == first).all()
