"""FP64 form: a prime that breaks off a stage (after interp_advance_deposit, before stage_temp) leaves the
primed RHS_T, whatever was bound when in the steps before: read back and stepped on, it equals a fresh
handle's that was given the same particles, bit for bit."""
import numpy as np
import pytest

import helpers
from first_repo_gb300 import gen, pstep

pytestmark = pytest.mark.gpu


def population(n, count, bp, seed):
    """away from the faces and slow: nothing wraps, so the base state a broken-off stage leaves is its start"""
    rng = np.random.default_rng(seed)
    x = bp.l * rng.uniform(0.2, 0.8, (3, count))
    v = 0.01 * rng.normal(size=(3, count))
    return [np.ascontiguousarray(a) for a in (*x, *v, 1.0 + 0.1 * rng.normal(size=count))]


@pytest.mark.parametrize("flags", [pstep.TRACK_ORDER | pstep.REFERENCE_SUMS, 0])
@pytest.mark.parametrize("stages", [0, 2])
def test_prime_that_breaks_off_a_stage(built_cuda, flags, stages):
    n, count = 12, 900
    bp = helpers.make_bp(n, count)
    fields = helpers.ghosted_fields(gen.make_case(n, 8, 5, False))

    def start(*arrs):
        g = pstep.ParticleStep(bp.step_config(), count, pstep.FP64, flags)
        g.load(*arrs)
        g.bind_velocity(*fields[:3])
        g.bind_temperature(fields[3])
        g.prime()
        return g

    g = start(*population(n, count, bp, 3), np.arange(count, dtype=np.int32))
    for k in range(4):  # a caller that binds the temperature between wrap and stage_temp
        g.interp_advance_deposit(k)
        g.wrap()
        g.bind_temperature(fields[3])
        g.stage_temp()
        g.end_stage()
    g.end_step()
    for k in range(stages):
        g.interp_advance_deposit(k)
        g.wrap()
        g.bind_temperature(fields[3])
        g.stage_temp()
        g.end_stage()
    g.interp_advance_deposit(stages)
    now = [np.empty(count) for _ in range(7)] + [np.empty(count, dtype=np.int32)]
    g.download(*now)
    g.prime()
    f = start(*now)
    assert g.max("RHS_T") == f.max("RHS_T")
    io, ig = np.argsort(f.array("flag")), np.argsort(g.array("flag"))
    assert helpers.bits_equal(g.array("RHS_T")[ig], f.array("RHS_T")[io])
    g.run(1)
    f.run(1)
    io, ig = np.argsort(f.array("flag")), np.argsort(g.array("flag"))
    for name in ("x", "u", "T", "RHS_T"):
        assert helpers.bits_equal(g.array(name)[ig], f.array(name)[io]), name
    assert g.check() == (0, 0) and f.check() == (0, 0)
    g.close()
    f.close()
