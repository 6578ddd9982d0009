"""The persistent forward kernel at the edges of its tiles and grid, and on tables that are only
4-byte aligned: a row's outputs depend on nothing but the row, so every call has to give, bit for
bit, what a call on the first 128 rows alone gives for them; and they are the bf16 network's, as
the oracle rounds it (the tolerance of tests/test_mlp_gpu.py: bf16 has 8 bits, activations O(1))."""
import ctypes as C

import numpy as np
import pytest

from first_repo_gb300 import mlp

pytestmark = pytest.mark.gpu


def rows(n, seed):
    return np.random.default_rng(seed).uniform(-1.0, 1.0, (n, mlp.N_IN)).astype(np.float32)


@pytest.mark.parametrize("n", [1, 127, 128, 129, 257, 4 * 152 * 256 + 1])
def test_rows_are_independent_of_the_call(built_cuda, n):
    net = mlp.Mlp(seed=3)
    x = rows(n, 4)
    y = net.forward(x)
    for at in {0, max(0, n - 128), max(0, n // 2 - 64)}:
        part = net.forward(x[at:at + 128])
        assert part.tobytes() == y[at:at + len(part)].tobytes()
    assert np.all(np.isfinite(y)) and (n == 1 or np.std(y) > 0)


@pytest.mark.parametrize("shift", [0, 1, 2])
def test_unaligned_device_tables(built_cuda, shift):
    import torch
    net = mlp.Mlp(seed=3)
    n = 300
    x = rows(n, 8)
    buf = torch.zeros(n * mlp.N_IN + 8, dtype=torch.float32, device="cuda")
    out = torch.zeros(n * mlp.N_OUT + 8, dtype=torch.float32, device="cuda")
    buf[shift:shift + n * mlp.N_IN] = torch.from_numpy(x.ravel()).cuda()
    torch.cuda.synchronize()
    net._check(net.L.pmlp_forward(net.h, C.c_void_p(buf.data_ptr() + 4 * shift), n,
                                  C.c_void_p(out.data_ptr() + 4 * shift), 1))
    got = out[shift:shift + n * mlp.N_OUT].cpu().numpy().reshape(n, mlp.N_OUT)
    assert got.tobytes() == net.forward(x).tobytes()
    assert not out[:shift].any() and not out[shift + n * mlp.N_OUT:].any()
