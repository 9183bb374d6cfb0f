"""The separable filters (csrc/sepfilter.cu) slab by slab: with the device's memory
taken but for less than the scratch of the whole grid, a step runs and gives the
fields of an unrestricted one (1e-13 relative: the same sums over the same
taps; a CTA's rows, and with them the scale of its integers, may differ)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gauss,leave", [(True, 64), (True, 12), (False, 40)])
def test_step_with_little_memory_left(built_lib, gauss, leave):
    import torch
    from exactclosure_gb300 import navierstokes as NS

    n, c, l = 150, 5, 1.0
    fdelta = NS.gaussian(l / n, 2 * l * c / n, 2) if gauss else None
    got = []
    for restricted in (False, True):
        d = NS.DnsAid(n, l, 2e-4, c, fdelta)
        d.init_random("power", -5 / 3, 1.0, 3)
        d.start()
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        fill = None
        if restricted:
            free = torch.cuda.mem_get_info()[0]
            fill = torch.empty(max(free - leave * 2**20, 0), dtype=torch.uint8, device="cuda")
        d.step(1.0, 0.4, max_steps=2)
        got.append({k: d.get(k) for k in NS.DNSAID_FIELDS} | {"u": d.velocity()})
        del fill
        torch.cuda.empty_cache()
        d.close()
    for k, a in got[0].items():
        assert np.linalg.norm(got[1][k] - a) <= 1e-13 * np.linalg.norm(a), k
