"""Chained launches (chain_wait): many small operators in a row on one stream,
on several streams and inside a captured graph give the bits of the same calls
one at a time with a synchronisation after each."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [4, 8, 24, 32, 44, 48])
def test_chained_calls_equal_single_calls(built_lib, n, precision):
    import torch

    from exactclosure_gb300 import navierstokes as NS

    dt = torch.float64 if precision == 0 else torch.float32
    g = NS.Grid(1.0, n)
    u0 = torch.randn((3, n, n, n), generator=torch.Generator("cuda").manual_seed(n), dtype=dt, device="cuda")

    def steps(ps, u, k, p, sync):
        for _ in range(12):
            for f in (lambda: NS.tensordivergence(k, u, 1e-3, g), lambda: NS.project(k, ps, p),
                      lambda: u.add_(k, alpha=1e-4)):
                f()
                if sync:
                    torch.cuda.synchronize()

    def run(sync, stream=None, graph=False):
        ps = NS.poissonsolver(g, precision)
        u, k, p = u0.clone(), torch.empty_like(u0), torch.empty_like(u0[0])
        torch.cuda.synchronize()
        with torch.cuda.stream(stream or torch.cuda.Stream()):
            if graph:
                cg = torch.cuda.CUDAGraph()
                with torch.cuda.graph(cg):
                    steps(ps, u, k, p, False)
                cg.replay()
            else:
                steps(ps, u, k, p, sync)
        return ps, u, k, p

    ref = run(True)
    torch.cuda.synchronize()
    others = [run(False), run(False), run(False, graph=True)]  # two streams at once, then a capture
    torch.cuda.synchronize()
    for o in others:
        for a, b in zip(ref[1:], o[1:]):
            assert torch.equal(a, b)
        o[0].close()
    ref[0].close()
