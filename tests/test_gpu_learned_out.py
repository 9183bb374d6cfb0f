"""The network's last layer writing the scaled fields (FP32, 64^3) and the
scaling in two floats: against the FP64 form of the same call, which packs and
unpacks with FP64 products -- equal up to the last rounding of a value (2^-23
relative), also for factors outside the floats' range and off 64^3."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scales", [(1.0, 1.0), (0.37, 41.3), (3.0e-25, 7.0e-22), (2.0, 1.0e30)])
@pytest.mark.parametrize("n,batch", [(64, 1), (64, 3), (16, 2), (12, 1)])
def test_float_fields_equal_the_double_ones(built_lib, n, batch, scales):
    import torch

    from exactclosure_gb300 import learned as LN

    net = LN.Net(7)
    net.set_scales(*scales)
    g = torch.Generator("cuda").manual_seed(n + batch)
    u = torch.randn((batch, 3, n, n, n), generator=g, device="cuda") * scales[0]
    m32, m64 = torch.empty_like(u), torch.empty(u.shape, dtype=torch.float64, device="cuda")
    net.forward(u, m32)
    net.forward(u.double(), m64)
    torch.cuda.synchronize()
    ref = m64.float()
    assert torch.isfinite(m32).all() and float(ref.abs().max()) > 0
    assert float(((m32 - ref).abs() / ref.abs().clamp_min(1e-37)).max()) <= 2.0**-23
    net.close()


@pytest.mark.parametrize("n", [16, 64])
def test_loss_and_gradients_of_both_types(built_lib, n):
    import torch

    from exactclosure_gb300 import learned as LN

    net = LN.Net(8)
    net.set_scales(0.7, 13.0)
    g = torch.Generator("cuda").manual_seed(n)
    u = torch.randn((2, 3, n, n, n), generator=g, device="cuda")
    m = torch.randn((2, 3, n, n, n), generator=g, device="cuda") * 13.0
    l32, g32 = net.gradients(u, m)
    l64, g64 = net.gradients(u.double(), m.double())
    assert abs(l32 - l64) <= 1e-6 * l64
    assert np.linalg.norm(g32 - g64) <= 1e-6 * np.linalg.norm(g64)
    net.close()
