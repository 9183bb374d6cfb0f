"""Projection and scalar solve of fields that start at an odd word: the register
passes of the FFT read pairs of words, so such a field takes the passes that read
words (csrc/fft.cu).  Grids with a compiled plan (32, 128: also the mixed solve)
and without one (30; 90: also the mixed solve), both precisions; against the
oracle at the tolerances of the plans' own tests, and the words around the
field stay as they were."""
import numpy as np
import pytest

from oracle import ns

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def NS(built_lib):
    from exactclosure_gb300 import navierstokes

    return navierstokes


def odd(a, dt):
    """A contiguous tensor of `a` one word into its buffer, and the buffer."""
    import torch

    buf = torch.full((a.size + 2,), 7.0, dtype=dt, device="cuda")
    return buf[1:-1].view(a.shape).copy_(torch.from_numpy(a)), buf


def rel(a, b):
    return float(np.linalg.norm((a - b).ravel()) / np.linalg.norm(b.ravel()))


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [30, 32, 90, 128])
def test_fields_at_an_odd_word(NS, n, precision):
    import torch

    dt, tol = (torch.float64, 1e-12) if precision == 0 else (torch.float32, 2e-5)
    u = np.random.default_rng(n).standard_normal((3, n, n, n))
    if precision:
        u = u.astype(np.float32).astype(np.float64)
    d = u[0] + 0.25
    if precision:
        d = d.astype(np.float32).astype(np.float64)
    ps = NS.poissonsolver(NS.Grid(1.0, n), precision)
    t, tb = odd(u, dt)
    p, pb = odd(np.zeros_like(d), dt)
    ps.project(t, p)
    ref, pref = ns.project(u, 1.0 / n, return_p=True)
    assert rel(t.double().cpu().numpy(), ref) < tol
    assert rel(p.double().cpu().numpy(), pref) < tol
    q, qb = odd(d, dt)
    ps.solve(q, q)
    assert rel(q.double().cpu().numpy(), ns.poisson_solve(d, 1.0 / n)) < tol
    for b in (tb, pb, qb):
        assert float(b[0]) == 7.0 and float(b[-1]) == 7.0
    ps.close()
