"""The one-pass scans (sort, order passes) do not depend on their waits: with a limit of one look at a
predecessor, and with none at all (every block sums what lies before its tile itself, through windows
of 32 tiles), a run gives what a run with the default limit gives, bit for bit, and no error."""
import numpy as np
import pytest

import helpers
from first_repo_gb300 import gen, pstep

pytestmark = pytest.mark.gpu


def run(n, count, precision, flags, wait):
    bp = helpers.make_bp(n, count)
    rng = np.random.default_rng(n)
    arrs = [np.ascontiguousarray(a) for a in
            (*(rng.uniform(0.0, bp.l, (3, count))), *(0.4 * bp.l / n / bp.dt * rng.uniform(-1.0, 1.0, (3, count))),
             1.0 + 0.1 * rng.normal(size=count))]
    fields = helpers.ghosted_fields(gen.make_case(n, 8, 5, False))
    g = pstep.ParticleStep(bp.step_config(), count, precision, flags)
    if wait:
        g.set_wait_limit(*wait)
    g.load(*arrs, np.arange(count, dtype=np.int32))
    g.bind_velocity(*fields[:3])
    g.bind_temperature(fields[3])
    g.prime()
    g.run(2)
    assert g.check() == (0, 0)
    at = np.argsort(g.array("flag")) if precision == pstep.FP32 else slice(None)
    out = [g.array(k)[at] for k in ("flag", "x", "y", "z", "u", "T", "RHS_T")] + [g.field(k) for k in pstep.FIELD_IDS]
    g.close()
    return out


# (42^3 keys: 19 tiles, 70000 particles: 3 tiles of bits; 64^3 keys: 64 tiles; one tile alone)
@pytest.mark.parametrize("n,count,precision,flags", [
    (40, 70001, pstep.FP64, pstep.TRACK_ORDER), (40, 70001, pstep.FP64, pstep.TRACK_ORDER | pstep.REFERENCE_SUMS),
    (64, 1001, pstep.FP64, pstep.TRACK_ORDER), (64, 30000, pstep.FP32, 0), (16, 500, pstep.FP32, 0),
    (8, 40, pstep.FP64, pstep.TRACK_ORDER)])
def test_results_do_not_depend_on_the_waits(built_cuda, n, count, precision, flags):
    want = run(n, count, precision, flags, None)
    for wait in ((1, False), (2, False), (0, True)):
        for a, b in zip(run(n, count, precision, flags, wait), want, strict=True):
            assert helpers.bits_equal(a, b), wait
