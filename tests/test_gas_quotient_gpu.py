"""The gas step's quotients (T = (P0 / R) / Rho_new) against a division, bit for bit: gas at rest keeps its
density through the first stage, so the stage's T is P0 / R over the density that was put in. Densities
over the whole range of doubles, zero, subnormal and infinite ones among them, each by itself in a
field of ones (what an infinite or missing density does to the rest of the stage is not looked at)."""
import numpy as np
import pytest

import pyoracle  # noqa: F401  (the oracle's path)
from first_repo_gb300 import gas
from test_gas_oracle import gas_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spread", [0.5, 30.0, 127.0, 300.0])
def test_temperature_is_the_division(built_cuda, spread):
    n = 16
    bp, _, _ = gas_case(n, 10, 21, cooling=1)  # P0 stays
    cfg = dict(bp.gas_config(), iterations=1)
    rng = np.random.default_rng(int(spread))
    rho = 10.0 ** rng.uniform(-spread, spread, (n, n, n))
    special = [0.0, 5e-324, 1e-310, 2.2250738585072014e-308, 1.7976931348623157e308, np.inf, 1.0, 2.0 ** -423,
               np.nextafter(2.0 ** 424, 0.0), 2.0 ** 424]
    if spread > 200:
        rho.ravel()[::97][:len(special)] = special
    zero = np.zeros((n, n, n))
    g = gas.GasStep(cfg)
    g.init(zero, zero, zero, rho)
    g.stage(0)
    inner = g.field("Rho_new")[1:-1, 1:-1, 1:-1]
    assert np.array_equal(inner, rho)
    with np.errstate(all="ignore"):
        want = (cfg["p0"] / (cfg["cp"] - cfg["cv"])) / rho
    got = g.field("T")[1:-1, 1:-1, 1:-1]
    assert np.array_equal(got, want), int((got != want).sum())
    g.close()
