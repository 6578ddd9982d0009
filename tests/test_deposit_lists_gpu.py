"""The FP64 brick deposit's lists at the lengths where their handling changes: empty nodes, one
thread's longest list (32), the first warp-summed one (33), segments at and past what the h-class
table holds (255), on a grid whose last bricks are ragged. Fields against the reference-order sums
(which equal the oracle bit for bit): the bound is the form's own 1e-12 of max|field|; a cell of N
particles rounds by about N 2^-53, 3e-13 at the largest here."""
import numpy as np
import pytest

import helpers
from first_repo_gb300 import gen, pstep

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("per_cell", [1, 32, 33, 255, 256, 2600])
@pytest.mark.parametrize("one_node", [False, True])
def test_dense_cells_match_reference_sums(built_cuda, per_cell, one_node):
    n = 13
    rng = np.random.default_rng(per_cell)
    # two full cells (one at the grid's far corner) and a sprinkle elsewhere
    count = 2 * per_cell + 40
    bp = helpers.make_bp(n, count)
    dx = bp.l / n
    off = rng.uniform(0.0, 1.0, (3, count))
    if one_node:
        off[:, :2 * per_cell] *= 0.49  # all of a cell's particles round to one node, one h class
    cell = rng.integers(0, n, (3, count)).astype(np.float64)
    cell[:, :per_cell] = np.array([[4.0], [7.0], [8.0]])
    cell[:, per_cell:2 * per_cell] = n - 1.0
    x = (cell + off) * dx
    vel = rng.normal(size=(3, count))
    t = 1.0 + 0.1 * rng.normal(size=count)
    case = gen.make_case(n, 8, 3, False)
    fields = helpers.ghosted_fields(case)
    got = {}
    for flags in (pstep.TRACK_ORDER, pstep.TRACK_ORDER | pstep.REFERENCE_SUMS):
        g = pstep.ParticleStep(bp.step_config(), count, pstep.FP64, flags)
        g.load(*[np.ascontiguousarray(a) for a in (*x, *vel, t)], np.arange(count, dtype=np.int32))
        g.bind_velocity(*fields[:3])
        g.bind_temperature(fields[3])
        g.prime()
        g.run(1)
        got[flags] = {k: g.field(k) for k in pstep.FIELD_IDS}
        g.close()
    a, b = got.values()
    for k in pstep.FIELD_IDS:
        assert helpers.max_rel_to_max(a[k], b[k]) <= 1e-12, k
