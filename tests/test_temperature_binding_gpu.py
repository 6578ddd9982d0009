"""FP64 form: where the stage's temperature gather runs (in the advance, or in stage_temp for a caller
that binds the temperature between the two) must not show: particles on cell faces, node edges and
wrapping positions, stage by stage, equal to the oracle bit for bit whatever the binding pattern,
also when RHS_T is asked for in mid-stage."""
import numpy as np
import pytest

import helpers
import pyoracle
from first_repo_gb300 import gen, pstep

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pattern", ["never", "always", "alternating", "asked"])
def test_binding_pattern_does_not_show(built_cuda, pattern):
    n, count = 12, 1500
    bp = helpers.make_bp(n, count)
    dx = bp.l / n
    rng = np.random.default_rng(9)
    x = rng.integers(0, 2 * n, (3, count)) * (0.5 * dx)  # on faces and node edges
    x[:, ::2] = rng.uniform(0.0, bp.l, (3, (count + 1) // 2))
    x[:, 1::5] = np.nextafter(x[:, 1::5], 10.0)
    x[:, 3::5] = np.maximum(np.nextafter(x[:, 3::5], -1.0), 0.0)
    x[0, 5] = 0.0
    x = np.minimum(x, np.nextafter(bp.l, 0.0))
    arrs = [np.ascontiguousarray(a) for a in (*x, *rng.normal(size=(3, count)), 1.0 + 0.1 * rng.normal(size=count))]
    arrs.append(np.arange(count, dtype=np.int32))
    fields = helpers.ghosted_fields(gen.make_case(n, 8, 5, False))
    o = pyoracle.Oracle(bp.step_config(), count)
    o.load(*arrs)
    o.prime(fields[3])
    g = pstep.ParticleStep(bp.step_config(), count, pstep.FP64, pstep.TRACK_ORDER | pstep.REFERENCE_SUMS)
    g.load(*arrs)
    g.bind_velocity(*fields[:3])
    g.bind_temperature(fields[3])
    g.prime()
    for step in range(2):
        o.run(1, *fields)
        for k in range(4):
            g.interp_advance_deposit(k)
            if pattern == "asked":
                g.array("RHS_T")
            g.wrap()
            if pattern == "always" or (pattern in ("alternating", "asked") and (step + k) % 2):
                g.bind_temperature(fields[3])
            g.stage_temp()
            g.end_stage()
        g.end_step()
        for name in ("x", "y", "z", "u", "v", "w", "T", "RHS_T"):
            assert helpers.bits_equal(g.array(name), o.array(name)), (step, name)
        assert helpers.bits_equal(g.field("RHS_Part_Temp"), o.fields["E"])
    assert g.check() == (0, 0)
    g.close()
