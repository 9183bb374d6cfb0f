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


@pytest.mark.parametrize("n", [16, 64])
@pytest.mark.parametrize("k", [112, 116])
def test_subnormal_weight_gradients(built_lib, n, k):
    """Targets 2^-k: the last layer's weight gradients, sums of products about
    2^-130, are those of targets of size one, scaled, but for the last bits of
    a subnormal number and of a BF16 gradient (one in 2^8 each; they cancel in a
    sum of n^3 random signs only to their own root mean square: a tenth)."""
    import torch
    from exactclosure_gb300 import learned as LN

    net = LN.Net(1)
    r = np.random.default_rng(0)
    p = [(r.normal(0, 0.1, (27, ci, co)).astype(np.float32), np.full(co, 0.0 if i == 2 else 2.0**-10, np.float32))
         for i, (ci, co) in enumerate(LN.VALID)]
    p[2] = (p[2][0] * 0, p[2][1])
    net.set_params(LN.flatten(p))
    g = torch.Generator("cuda").manual_seed(1)
    u = torch.randn((1, 3, n, n, n), generator=g, device="cuda") * 2.0**-10
    m = torch.randn((1, 3, n, n, n), generator=g, device="cuda")
    if n == 64:
        k -= 12  # a voxel's gradient has the factor 2 / (3 n^3)
    big, small = (np.float64(LN.unflatten(net.gradients(u, m * 2.0**-e)[1])[2][0]) * 2.0**e for e in (0, k))
    assert np.linalg.norm(big) > 0
    assert np.linalg.norm(small - big) < 0.1 * np.linalg.norm(big)
    net.close()
