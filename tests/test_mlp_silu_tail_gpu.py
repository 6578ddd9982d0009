"""The activation z sigmoid(z) where the sigmoid is below the smallest normal number (z from -87.3 down to
-88.7, where exp(-z) leaves fp32), through a network that hands one input to the output: two layers
with one unit weight each and an identity in between are silu(silu(x)), and the inner value's bf16 is
seen through the outer silu, which halves numbers this small. bf16 reaches down to 9e-41, so nothing
of this is lost to the format: the bound is one bf16 step of each rounding (2^-8 of the value, three of
them) and one of the sigmoid's subnormal steps (1.4e-45) times |z|. Below, the result is 0."""
import numpy as np
import pytest

from first_repo_gb300 import mlp

pytestmark = pytest.mark.gpu


def test_activation_below_the_normal_range(built_cuda):
    net = mlp.Mlp(seed=1)
    p = np.zeros_like(net.params)
    hid, inp = 64, 16
    o_b1, o_w2 = hid * inp, hid * inp + hid
    o_w3 = o_w2 + hid * hid + hid
    p[5 * inp + 2] = 1.0          # hidden 5 <- input 2
    p[o_b1 + 5] = -80.0           # its bias carries z there in steps finer than bf16's
    p[o_w2 + 9 * hid + 5] = 1.0   # hidden 9 <- hidden 5
    p[o_w3 + 1 * hid + 9] = 1.0   # output 1 <- hidden 9
    net.params = p
    x = np.zeros((1000, mlp.N_IN), dtype=np.float32)
    steps = np.arange(1000) % 256
    x[:, 2] = -6.0 - steps / 64.0  # bf16 numbers from -6 to -10 (eight bits: in steps of 1/32 from -8 on)
    import torch
    z = torch.from_numpy(x[:, 2]).to(torch.bfloat16).to(torch.float64).numpy() - 80.0
    y = net.forward(x)[:, 1].astype(np.float64)
    with np.errstate(over="ignore"):
        inner = z / (1.0 + np.exp(-z))
    want = 0.5 * inner
    live = z >= -88.7
    assert np.count_nonzero(live & (z < -87.4)) > 50
    assert np.all(np.abs(y - want)[live] <= 3 * 2.0 ** -8 * np.abs(want[live]) + 89 * 1.4e-45)
    assert np.all(y[z < -88.75] == 0.0)
