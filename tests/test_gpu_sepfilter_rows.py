"""The x pass of the separable filters (csrc/sepfilter.cu) where eight rows and
their ghosts are exactly the 48 KB of shared memory a launch has by default: DNS
750^3 with ratio 5 and the reference's Gaussian (nine ghosts on either side),
which leaves no room for the kernel's static words.  One step; the exact
closure keeps its LES on the filtered DNS: 1e-12 relative, as in the small
grids' tests."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_rows_that_fill_the_shared_memory(built_lib):
    from exactclosure_gb300 import navierstokes as NS

    n, c, l = 750, 5, 1.0
    d = NS.DnsAid(n, l, 2e-4, c, NS.gaussian(l / n, 2 * l * c / n, 2))
    d.init_random("power", -5 / 3, 1.0, 1)
    d.start()
    assert d.step(1.0, 0.4, max_steps=1) == 1
    e = d.errors()
    assert np.isfinite(list(e.values())).all()
    assert e["u_cfd"] < 1e-12 and e["u_nomo"] > 1e-8, e
    d.close()
