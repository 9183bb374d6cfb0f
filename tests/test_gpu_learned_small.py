"""The network's scaling in two floats (csrc/learned.cu) where the product with the
factor's low part would underflow: outputs about 2^-126 equal the rounded FP64
products of the same call with FP64 fields, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [16, 64])
@pytest.mark.parametrize("exponent", [-62, -48, -20])
def test_small_outputs_round_like_fp64(built_lib, n, exponent):
    import torch
    from exactclosure_gb300 import learned as LN

    net = LN.Net(5)
    net.set_scales(1.0, 1.1 * 2.0**-60)
    p = LN.unflatten(net.get_params())
    net.set_params(LN.flatten(p[:2] + [(p[2][0] * np.float32(2.0**exponent), p[2][1] * np.float32(2.0**exponent))]))
    u = torch.randn((1, 3, n, n, n), generator=torch.Generator("cuda").manual_seed(n), device="cuda")
    m32, m64 = torch.empty_like(u), torch.empty(u.shape, dtype=torch.float64, device="cuda")
    net.forward(u, m32)
    net.forward(u.double(), m64)
    assert float(m64.abs().max()) > 0
    assert torch.equal(m32, m64.float())
    net.close()
