"""The order within a node at the segment lengths where its sorting changes hands: ranked items (up
to 128), the 16 KB bitonic sort (up to 2048), the 128 KB one (up to 16384). In reference order the
deposited fields and the particle order have to equal the oracle's bit for bit, which only the
exact order of every segment gives."""
import numpy as np
import pytest

import helpers
import pyoracle
from first_repo_gb300 import gen, pstep

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("per_node", [2, 128, 129, 2048, 2049, 5000])
def test_long_segments_equal_the_oracle(built_cuda, per_node):
    n, rest = 8, 37
    count = per_node + rest
    bp = helpers.make_bp(n, count)
    dx = bp.l / n
    rng = np.random.default_rng(per_node)
    x = (rng.uniform(-0.45, 0.45, (3, count)) + 3.0) * dx  # all round to one node, every h class
    x[:, per_node:] = rng.uniform(0.0, bp.l, (3, rest))
    x = x[:, rng.permutation(count)]
    vel = 0.1 * rng.normal(size=(3, count))
    arrs = [np.ascontiguousarray(a) for a in (*x, *vel, 1.0 + 0.1 * rng.normal(size=count))]
    arrs.append(np.arange(count, dtype=np.int32))
    fields = helpers.ghosted_fields(gen.make_case(n, 8, 5, False))
    o = pyoracle.Oracle(bp.step_config(), count)
    o.load(*arrs)
    o.prime(fields[3])
    o.run(1, *fields)
    g = pstep.ParticleStep(bp.step_config(), count, pstep.FP64, pstep.TRACK_ORDER | pstep.REFERENCE_SUMS)
    g.load(*arrs)
    g.bind_velocity(*fields[:3])
    g.bind_temperature(fields[3])
    g.prime()
    g.run(1)
    assert g.check() == (0, 0)
    assert helpers.bits_equal(g.array("flag"), o.flag())
    for ours, theirs in (("C", "C"), ("RHS_RU_x", "Ax"), ("RHS_RU_z", "Az"), ("RHS_Part_Temp", "E")):
        assert helpers.bits_equal(g.field(ours), o.fields[theirs]), ours
    g.close()
