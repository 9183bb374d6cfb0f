"""Handles of FP64 grids without a compiled FFT plan where the device's memory is
nearly taken: what the mixed-precision solve and the batched LES solves hold
beyond the plain passes is left out, and the handle is made all the same, with
results to rounding of those of an unrestricted one (1e-12)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def NS(built_lib):
    from exactclosure_gb300 import navierstokes

    return navierstokes


class Taken:
    """All of the device's memory but `leave` MiB."""

    def __init__(self, leave):
        self.leave = leave

    def __enter__(self):
        import torch

        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        self.t = torch.empty(torch.cuda.mem_get_info()[0] - self.leave * 2**20, dtype=torch.uint8, device="cuda")

    def __exit__(self, *a):
        import torch

        del self.t
        torch.cuda.empty_cache()


def held(make):
    """MiB that make()'s handle takes, and the handle."""
    import torch

    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    a = torch.cuda.mem_get_info()[0]
    h = make()
    torch.cuda.synchronize()
    return (a - torch.cuda.mem_get_info()[0]) // 2**20, h


def close_to(a, b):
    return np.linalg.norm(a - b) <= 1e-12 * np.linalg.norm(b)


def test_solver(NS):
    import torch

    n = 250
    u = torch.randn((3, n, n, n), generator=torch.Generator("cuda").manual_seed(0), dtype=torch.float64, device="cuda")
    v = u.clone()
    mib, ps = held(lambda: NS.poissonsolver(NS.Grid(1.0, n)))
    ps.project(u)
    ps.close()
    with Taken(mib - 100):  # the mixed solve holds 20 bytes a cell: 300 MiB
        ps = NS.poissonsolver(NS.Grid(1.0, n))
    ps.project(v)
    ps.close()
    assert float((u - v).norm()) <= 1e-12 * float(u.norm())


def test_case(NS):
    out = []
    make = lambda: NS.Case(180, 1.0, 1 / 2000, 0.3, les=[(2, "volume"), (2, "face")])
    mib, cs = held(make)
    for restricted in (False, True):
        if restricted:
            with Taken(mib - 60):  # 20 bytes a cell of the DNS and of both LES: 150 MiB
                cs = make()
        cs.init_random(4.0, 1.0, 0)
        cs.step(2)
        out.append([cs.velocity()] + [cs.les(i, w) for i in range(2) for w in ("exact", "nomodel")])
        cs.close()
    for a, b in zip(*out):
        assert close_to(b, a)


def test_euler_driver(NS):
    out = []
    make = lambda: NS.DnsAid(150, 1.0, 2e-4, 3)
    mib, d = held(make)
    for restricted in (False, True):
        if restricted:
            with Taken(mib - 40):
                d = make()
        d.init_random("power", -5 / 3, 1.0, 3)
        d.start()
        d.step(1.0, 0.4, max_steps=1)
        out.append([d.velocity()] + [d.get(k) for k in NS.DNSAID_FIELDS])
        d.close()
    for a, b in zip(*out):
        assert close_to(b, a)
