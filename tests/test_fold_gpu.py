"""The ghost fold, refresh and interior sums in one launch, at the smallest grids (every cell a
corner, one interior cell a dimension), a ragged one and one with more rows than the launch's
warps. The folded and refreshed fields equal the oracle's bit for bit, ghosts included; the sums
have an order of their own: within 1e-12 of the sum of magnitudes (N additions round by at most
N 2^-53 of it when added in one chain, 130^3 x 2^-53 = 2.4e-10, but a tree of chains of at most
(130 / 32 + 1) x 3 + 8 + 4 + 8 additions by 40 x 2^-53)."""
import numpy as np
import pytest

import helpers
import pyoracle
from first_repo_gb300 import gen, pstep

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, twc", [(2, 1), (2, 0), (3, 1), (17, 1), (33, 0), (130, 1)])
def test_fold_matches_oracle(built_cuda, n, twc):
    count = 4000
    bp = helpers.make_bp(n, count, {"twc": twc})
    cfg = bp.step_config()
    case = gen.make_case(n, count, n, False)
    arrays = [np.ascontiguousarray(case[k]) for k in ("x", "y", "z", "u", "v", "w", "t", "flag")]
    ux, uy, uz, tf = helpers.ghosted_fields(case)
    o = pyoracle.Oracle(cfg, count)
    o.load(*arrays)
    o.prime(tf)
    g = pstep.ParticleStep(cfg, count, pstep.FP64, pstep.TRACK_ORDER | pstep.REFERENCE_SUMS)
    g.load(*arrays)
    g.bind_velocity(ux, uy, uz)
    g.bind_temperature(tf)
    g.prime()
    for k in range(2):
        o.stage(k, ux, uy, uz, tf)
        g.stage(k)
        for f, name in helpers.FIELD_MAP.items():
            assert helpers.bits_equal(g.field(name), o.fields[f]), (k, f)
        E = o.fields["E"][1:-1, 1:-1, 1:-1]
        assert abs(g.energy_mean() - E.mean()) <= 1e-12 * np.abs(E).mean()
        got = g.momentum_sums()
        for d, f in enumerate(("Ax", "Ay", "Az")):
            a = o.fields[f][1:-1, 1:-1, 1:-1]
            assert abs(got[d] - a.sum()) <= 1e-12 * np.abs(a).sum()
        o.end_stage()
        g.end_stage()
    g.close()
