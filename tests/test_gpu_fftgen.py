"""The run-time register plans (csrc/fftgen.cuh) where their passes can go
wrong: line lengths with a factor of one, prime and square factors, the largest
radix, tiles and row blocks that do not divide the grid, the first grid of the
mixed-precision solve and the last before it -- the projection and the scalar
solve against the oracle, in both precisions and every engine.  Tolerances are
those of the compiled plans' tests: 1e-12 relative L2 in FP64, 2e-5 in FP32."""
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


@pytest.mark.parametrize("precision,engine", [(0, 0), (0, 2), (1, 0), (1, 2)])
@pytest.mark.parametrize("n", [4, 6, 10, 14, 22, 26, 34, 36, 50, 66, 80, 84, 98, 110, 170, 204])
def test_projection_and_scalar_solve(NS, n, precision, engine):
    import torch

    dt, tol = (torch.float64, 1e-12) if precision == 0 else (torch.float32, 2e-5)
    u = np.random.default_rng(n).standard_normal((3, n, n, n))
    t = torch.from_numpy(u).cuda().to(dt)
    u = t.double().cpu().numpy()
    ps = NS.poissonsolver(NS.Grid(1.0, n), precision, engine)
    p = torch.empty_like(t[0])
    ps.project(t, p)
    ref, pref = ns.project(u, 1.0 / n, return_p=True)
    assert rel(t.double().cpu().numpy(), ref) < tol
    assert rel(p.double().cpu().numpy(), pref) < tol
    d = torch.from_numpy(u[0] + 0.25).cuda().to(dt)
    ref = ns.poisson_solve(d.double().cpu().numpy(), 1.0 / n)
    q = torch.empty_like(d)
    ps.solve(q, d)
    assert rel(q.double().cpu().numpy(), ref) < tol
    ps.solve(d, d)  # the right-hand side may be the output
    assert (d == q).all()
    ps.close()


@pytest.mark.parametrize("n", [250, 486])
def test_large_factors_match_stockham(NS, n):
    import torch

    g = torch.Generator(device="cuda").manual_seed(n)
    u = torch.randn((3, n, n, n), dtype=torch.float64, device="cuda", generator=g)
    out = []
    for engine in (0, 1):
        ps = NS.poissonsolver(NS.Grid(1.0, n), 0, engine)
        t, p = u.clone(), torch.empty_like(u[0])
        ps.project(t, p)
        out.append((t, p))
        ps.close()
    for a, b in zip(*out):
        assert float((a - b).norm() / b.norm()) < 1e-12


@pytest.mark.parametrize("precision", [0, 1])
def test_served_batch_equals_the_case(NS, built_lib, precision):
    """Several slots of one run-time-planned grid (the batched passes)."""
    from exactclosure_gb300.serving import Server

    n, steps = 50, 6
    sv = Server(precision=precision, autotune=False, slots_per_chunk=3)
    ids = [sv.submit(n, 1 / 2000, steps, seed=s, keep_field=True) for s in range(3)]
    sv.drain()
    got = {r["id"]: r["field"] for r in sv.poll()}
    for s, i in enumerate(ids):
        cs = NS.Case(n, 1.0, 1 / 2000, 0.3, precision=precision)
        cs.init_random(4.0, 1.0, s)
        cs.step(steps)
        assert (cs.velocity() == got[i]).all()
        cs.close()
    sv.close()


@pytest.mark.parametrize("e", [-900, -300, -130, -70, -40, 60, 100, 140, 400])
def test_mixed_solve_beyond_the_floats(NS, e):
    """A solve is linear: inputs scaled by 2^e, far outside FP32's exponents too,
    give the scaled results to 1e-12."""
    import torch

    n = 84
    gen = torch.Generator("cuda").manual_seed(3)
    u = torch.randn((3, n, n, n), generator=gen, dtype=torch.float64, device="cuda")
    d = torch.randn((n, n, n), generator=gen, dtype=torch.float64, device="cuda")
    d -= d.mean()
    ps = NS.poissonsolver(NS.Grid(1.0, n), 0)
    out = []
    for k in (0, e):
        a, p, q = u * 2.0**k, torch.empty_like(d), torch.empty_like(d)
        ps.project(a, p)
        ps.solve(q, d * 2.0**k)
        out.append([x * 2.0**-k for x in (a, p, q)])
    for x, y in zip(*out):
        assert float((x - y).norm() / x.norm()) < 1e-12
    ps.close()
