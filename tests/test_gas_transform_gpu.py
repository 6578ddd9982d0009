"""The gas step's Poisson transforms over every line count and tile width that its sizes choose (widths of
16, 9 .. 15, 5 and 3 bins along y, eight and four lines a CTA, more than 48 KB of shared memory), by the
solve itself: with uniform density and a velocity that is free of divergence to the last bit the density stays
1, and one iteration's pressure is the spectral solution of the discrete Poisson equation for the
right-hand side formed from the stage's own velocity and divergence. Against torch's transform in 64 bits: a
transform of n^3 points rounds by a few times log2(n^3) 2^-53 of its largest value, 3e-15 here; the smallest
wavenumber's division multiplies nothing, so the bound is 1e-12 of max|P|."""
import math

import numpy as np
import pytest
import torch

import helpers
import pyoracle  # noqa: F401  (the oracle's path)
from first_repo_gb300 import gas

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [8, 16, 32, 64, 128, 256, 512])
def test_one_solve_is_the_spectral_solution(built_cuda, n):
    bp = helpers.make_bp(n, 10)
    bp.cooling = 1
    bp.mu0 = min(bp.mu0, 0.05 * (bp.l / n) ** 2 / bp.dt)
    cfg = dict(bp.gas_config(), iterations=1)
    rng = np.random.default_rng(n)
    plane = rng.normal(size=(3, n, n))
    ru = [np.ascontiguousarray(np.broadcast_to(p, (n, n, n))) for p in
          (plane[0][:, :, None], plane[1][:, None, :], plane[2][None, :, :])]  # [z, y, x]: x, y, z not in each
    g = gas.GasStep(cfg)
    g.init(*ru, np.ones((n, n, n)))
    del ru
    g.stage(0)
    assert g.iterations() == 1

    def field(name):
        f = torch.empty((n + 2,) * 3, dtype=torch.float64, device="cuda")
        g.field_to(name, f.data_ptr())
        torch.cuda.synchronize()
        return f

    rho = field("Rho_new")
    assert bool((rho == 1.0).all())
    del rho
    dx = bp.l / n
    rhs = -field("divergence")[1:-1, 1:-1, 1:-1]
    inner, up = slice(1, -1), slice(2, None)
    u = field("U_x")
    rhs += (u[inner, inner, up] - u[inner, inner, inner]) / dx
    u = field("U_y")
    rhs += (u[inner, up, inner] - u[inner, inner, inner]) / dx
    u = field("U_z")
    rhs += (u[up, inner, inner] - u[inner, inner, inner]) / dx
    del u
    rhs /= cfg["dt"] * 0.5
    rhs -= rhs.mean()
    k = torch.arange(n, dtype=torch.float64, device="cuda")
    wave = 2.0 / dx ** 2 * (1.0 - torch.cos(2.0 * math.pi * k / n))
    spec = torch.fft.rfftn(rhs)
    den = wave[:, None, None] + wave[None, :, None] + wave[None, None, :n // 2 + 1]
    den[0, 0, 0] = 1.0
    spec /= -den
    want = torch.fft.irfftn(spec, s=(n, n, n))
    got = field("P")[1:-1, 1:-1, 1:-1]
    top = float(want.abs().max())
    assert top > 0.0
    assert float((got - want).abs().max()) <= 1e-12 * top
    g.close()
