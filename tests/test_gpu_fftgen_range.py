"""The mixed-precision solve on run-time plans (csrc/fftgen.cuh) between the
right-hand sides whose three corrections stay within the floats as they are and
those beyond the first one: scaled by 2^e the results scale, to the accuracy of
a solve in range.  Tolerance 4e-15: both results are within a few 2^-53 of the
exact one (1.1e-15 measured for FP64 transforms of the same grid)."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("e", [-66, -63, 84, 90])
@pytest.mark.parametrize("n", [84, 90])
def test_three_corrections(built_lib, n, e):
    import torch

    from exactclosure_gb300 import navierstokes as NS

    g = torch.Generator("cuda").manual_seed(n)
    u = torch.randn((3, n, n, n), generator=g, dtype=torch.float64, device="cuda")
    d = u[0] - u[0].mean()
    ps = NS.poissonsolver(NS.Grid(1.0, n), 0)
    out = []
    for k in (0, e):
        a, p, q = u * 2.0**k, torch.empty_like(d), torch.empty_like(d)
        ps.project(a, p)
        # the scalar solve's right-hand side is h d inside
        ps.solve(q, d * 2.0**k)
        out.append([x * 2.0**-k for x in (a, p, q)])
    for x, y in zip(*out):
        assert float((x - y).norm() / x.norm()) < 4e-15
    ps.close()
