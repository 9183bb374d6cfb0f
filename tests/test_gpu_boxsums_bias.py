"""The integer box sums (csrc/filter.cu, sum_fixed) of values over many binades: the
error of the filtered field has no mean.  Ratio 4: the weights are powers of
two, so a filtered value has the roundings of five sums of sixteen, of their
scaling (none) and of four additions, each to nearest: at most half a unit of
2^-53 of the value, 0.29 in the root mean square, independent -- 0.9 units, and 0.018
in the mean over 41472 values at four standard deviations."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_filtered_field_is_not_biased(built_lib):
    import torch
    from exactclosure_gb300 import navierstokes as NS

    n, c = 96, 4
    m = n // c
    u = np.exp(3 * np.random.default_rng(0).standard_normal((3, n, n, n)))
    cs = NS.Case(n, 1.0, 1 / 2000, 0.3, les=[(c, "face")])
    cs.set_velocity(u)
    cs.step(1)
    pair = torch.empty((2, 3, m, m, m), dtype=torch.float64, device="cuda")
    cs.snapshot(0, pair[0], pair[1])
    got = pair[0].cpu().numpy()
    cs.close()
    mean = 0.0
    for i in range(3):
        v = u[i].astype(np.longdouble)
        ax = 2 - i
        v = np.take(v, np.arange(m) * c + c - 1, axis=ax)  # the face: a point along its own axis
        for a in range(3):
            if a != ax:
                v = v.reshape(v.shape[:a] + (m, c) + v.shape[a + 1:]).sum(axis=a + 1)
        ref = v / 16
        mean += float(((got[i] - ref) / ref).mean()) * 2.0**53 / 3
    assert abs(mean) < 0.02, mean
