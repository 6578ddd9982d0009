"""The order passes at the sizes where their handling changes: one particle, around a bitmap word
and a 16-byte group of leave codes, more than one scan tile (32,768 positions), more leavers than
the pass kernel's threads (8,192); with no, few, half and all particles leaving. The particles' order
after every stage is the oracle's, exactly."""
import numpy as np
import pytest

import helpers
import pyoracle
from first_repo_gb300 import gen, pstep

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 16, 31, 33, 1000, 40001])
@pytest.mark.parametrize("share", [0.0, 0.01, 0.5, 1.0])
def test_order_matches_oracle(built_cuda, count, share):
    n = 8
    rng = np.random.default_rng(count + int(100 * share))
    bp = helpers.make_bp(n, count)
    cfg = bp.step_config()
    # the leaving ones start at a face and move out of it, the others stay near the middle
    x = bp.l * rng.uniform(0.4, 0.6, (3, count))
    vel = 0.01 * bp.l * rng.normal(size=(3, count))
    side = rng.integers(-1, 2, (3, count))
    out = rng.uniform(size=count) < share
    speed = 2.0 * bp.l / n
    x = np.where(out & (side != 0), np.where(side > 0, bp.l - 1e-6 * bp.l, 1e-6 * bp.l), x)
    vel = np.where(out, side * speed, vel)
    t = 1.0 + 0.1 * rng.normal(size=count)
    arrays = [np.ascontiguousarray(a) for a in (*x, *vel, t)] + [np.arange(count, dtype=np.int32)]
    ux, uy, uz, tf = helpers.ghosted_fields(gen.make_case(n, 8, 3, False))
    o = pyoracle.Oracle(cfg, count)
    o.load(*arrays)
    o.prime(tf)
    g = pstep.ParticleStep(cfg, count, pstep.FP64, pstep.TRACK_ORDER)
    g.load(*arrays)
    g.bind_velocity(ux, uy, uz)
    g.bind_temperature(tf)
    g.prime()
    for s in range(2):
        for k in range(4):
            o.stage(k, ux, uy, uz, tf)
            g.stage(k)
            assert np.array_equal(g.array("flag"), o.flag()), (s, k)
            assert helpers.bits_equal(g.array("x_new"), o.array("x_new")), (s, k)
            o.end_stage()
            g.end_stage()
        o.end_step()
        g.end_step()
    assert g.check() == (0, 0)
    g.close()
