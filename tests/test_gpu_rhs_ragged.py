"""FP32 right-hand side of rows that are multiples of four and no multiple of
the 64-cell tile: the 2 x 2 kernel's ragged tiles give the bits of the general
kernel (taken for fields that are not 16-byte aligned), and the oracle's values
(2e-5 relative L2, the FP32 operators' bound)."""
import numpy as np
import pytest

from oracle import ns

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("doadd", [False, True])
@pytest.mark.parametrize("n", [72, 84, 88, 96, 100, 132, 180, 196, 260, 324])
def test_ragged_tiles_equal_the_general_kernel(built_lib, n, doadd):
    import torch

    from exactclosure_gb300 import navierstokes as NS

    g, N = NS.Grid(1.0, n), 3 * n**3
    gen = torch.Generator("cuda").manual_seed(n)
    u = torch.randn(N, generator=gen, device="cuda")
    o = torch.randn(N, generator=gen, device="cuda")
    u1 = torch.empty(N + 1, device="cuda")[1:]
    o1 = torch.empty(N + 1, device="cuda")[1:]
    u1.copy_(u)
    o1.copy_(o)
    shape = (3, n, n, n)
    NS.tensordivergence(o.view(shape), u.view(shape), 1e-3, g, doadd)
    NS.tensordivergence(o1.view(shape), u1.view(shape), 1e-3, g, doadd)
    assert torch.equal(o, o1)
    if n <= 100 and not doadd:
        ref = ns.rhs(u.view(shape).double().cpu().numpy(), 1e-3, 1.0 / n)
        got = o.view(shape).double().cpu().numpy()
        assert np.linalg.norm(got - ref) < 2e-5 * np.linalg.norm(ref)


def test_served_slots_equal_the_case(built_lib):
    from exactclosure_gb300 import navierstokes as NS
    from exactclosure_gb300.serving import Server

    n, steps = 84, 3
    sv = Server(precision=1, autotune=False, slots_per_chunk=4)
    ids = [sv.submit(n, 1 / 500, steps, seed=s, keep_field=True) for s in range(4)]
    sv.drain()
    got = {r["id"]: r["field"] for r in sv.poll()}
    for s, i in enumerate(ids):
        cs = NS.Case(n, 1.0, 1 / 500, 0.3, precision=1)
        cs.init_random(4.0, 1.0, s)
        cs.step(steps)
        assert (cs.velocity() == got[i]).all()
        cs.close()
    sv.close()
