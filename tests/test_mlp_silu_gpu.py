"""The activation z sigmoid(z) over its range, through a network that hands one input on: with W1,
W2 and W3 one unit weight each the output is silu(silu(x)) with bf16 roundings between the layers.
Against the same in 64 bits: fp32 values that are right to an ulp or two (2^-22) round to another
bf16 value for about one in 2^13, and then by one bf16 step (2^-7 of the value at most); below
z = -87 the result may be flushed, |y| < 1.1e-36."""
import numpy as np
import pytest
import torch

from first_repo_gb300 import mlp

pytestmark = pytest.mark.gpu


def bf16(a):
    return torch.from_numpy(np.asarray(a, dtype=np.float32)).to(torch.bfloat16).to(torch.float64).numpy()


def silu(z):
    with np.errstate(over="ignore"):
        return z / (1.0 + np.exp(-z))


@pytest.mark.parametrize("top", [1e-3, 1.0, 20.0, 90.0, 1e30])
def test_activation_over_its_range(built_cuda, top):
    net = mlp.Mlp(seed=1)
    p = np.zeros_like(net.params)
    hid, inp, outp = 64, 16, 16
    o_w1, o_w2 = 0, hid * inp + hid
    o_w3 = o_w2 + hid * hid + hid
    p[o_w1 + 5 * inp + 2] = 1.0   # hidden 5 <- input 2
    p[o_w2 + 9 * hid + 5] = 1.0   # hidden 9 <- hidden 5
    p[o_w3 + 1 * hid + 9] = 1.0   # output 1 <- hidden 9
    net.params = p
    x = np.zeros((20001, mlp.N_IN), dtype=np.float32)
    x[:, 2] = bf16(np.linspace(-top, top, len(x)))
    y = net.forward(x)
    want = bf16(silu(bf16(silu(x[:, 2].astype(np.float64)))))
    got = y[:, 1].astype(np.float64)
    assert np.all(np.isfinite(got)) and not y[:, [0, 2, 3]].any()
    off = np.abs(got - want)
    assert np.all(off <= np.maximum(2.0 ** -7 * np.abs(want), 1.1e-36))
    assert np.mean(off > 1.1e-36) <= 2.0 ** -9
