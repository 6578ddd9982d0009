"""The gas step over the sizes its transforms tile differently (8 to 128: one partial bin tile, odd
half spectra, every line count) and with every source term on, against the C restatement: the bound
is the gas step's own 1e-10 of each field's range after the steps (tests/test_gas_gpu.py)."""
import numpy as np
import pytest

import pyoracle
from first_repo_gb300 import gas
from test_gas_gpu import _rel
from test_gas_oracle import gas_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [8, 16, 64, 128])
def test_all_terms_match_restatement(built_cuda, n):
    bp, fields, _ = gas_case(n, 10, 21)
    cfg = dict(bp.gas_config(), a_force=0.3, u0=0.2, gx=0.1, gy=-0.2, gz=0.4)
    o = pyoracle.GasOracle(cfg, None)
    g = gas.GasStep(cfg)
    args = [fields[k] for k in ("RU_x", "RU_y", "RU_z", "Rho")]
    o.init(*args, cfg["p0"])
    g.init(*args)
    for _ in range(2 if n < 128 else 1):
        o.step()
        g.step()
    for k in ("RU_x", "RU_y", "RU_z", "Rho", "P", "T", "U_x", "U_y", "U_z", "divergence", "Rho_new", "RHS_RU_x",
              "RHS_RU_y", "RHS_RU_z"):
        assert _rel(g.field(k), o.field(k)) <= 1e-10, (k, _rel(g.field(k), o.field(k)))
        f = g.field(k)  # the ghost layers are the periodic images
        assert np.array_equal(f[0], f[-2]) and np.array_equal(f[:, -1], f[:, 1]) and np.array_equal(f[:, :, 0], f[:, :, -2])
    assert abs(g.p0() - o.p0()) <= 1e-14
