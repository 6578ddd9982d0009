"""The reference-order deposit, where a warp merges the node lists around 4 x 4 x 2 targets 32
particles at a time: grids with every remainder of the target blocks, and as many particles in
two neighbouring cells as just miss, fill and pass one and two rounds, with and without the
momentum deposits. Every field equals the oracle's bit for bit: the additions and their order are
the same."""
import numpy as np
import pytest

import helpers
import pyoracle
from first_repo_gb300 import gen, pstep

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, per_cell, twc", [(4, 31, 1), (5, 32, 1), (6, 33, 1), (7, 63, 1), (8, 64, 0), (9, 65, 1),
                                              (10, 1, 1), (11, 500, 0)])
def test_rounds_and_ragged_blocks_match_oracle(built_cuda, n, per_cell, twc):
    rng = np.random.default_rng(100 * n + per_cell)
    count = 2 * per_cell + 30
    bp = helpers.make_bp(n, count, {"twc": twc})
    dx = bp.l / n
    cell = rng.integers(0, n, (3, count)).astype(np.float64)
    cell[:, :per_cell] = np.array([[1.0], [2.0], [3.0]])
    cell[:, per_cell:2 * per_cell] = np.array([[2.0], [2.0], [3.0]])
    x = (cell + rng.uniform(0.01, 0.99, (3, count))) * dx
    x = x[:, rng.permutation(count)]  # the two cells' lists alternate in the reference's order
    vel = rng.normal(size=(3, count))
    t = 1.0 + 0.1 * rng.normal(size=count)
    arrays = [np.ascontiguousarray(a) for a in (*x, *vel, t)] + [np.arange(count, dtype=np.int32)]
    ux, uy, uz, tf = helpers.ghosted_fields(gen.make_case(n, 8, 3, False))
    cfg = bp.step_config()
    o = pyoracle.Oracle(cfg, count)
    o.load(*arrays)
    o.prime(tf)
    g = pstep.ParticleStep(cfg, count, pstep.FP64, pstep.TRACK_ORDER | pstep.REFERENCE_SUMS)
    g.load(*arrays)
    g.bind_velocity(ux, uy, uz)
    g.bind_temperature(tf)
    g.prime()
    for k in range(4):
        o.stage(k, ux, uy, uz, tf)
        g.stage(k)
        for f, name in helpers.FIELD_MAP.items():
            assert helpers.bits_equal(g.field(name), o.fields[f]), (k, f)
        o.end_stage()
        g.end_stage()
    g.close()
