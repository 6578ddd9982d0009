"""FP64 form: a stage's temperature is the one bound when interp_advance_deposit ran unless another is bound
before stage_temp, whatever the caller did in earlier stages. Two handles over one population take the
same calls but for a first step in which only one of them binds the (same) temperature again between
wrap and stage_temp, after which its advances leave the gather to stage_temp. In the next stage
another field is bound, the device field is overwritten in place, or the heat-transfer coefficient is
changed; RHS_T, asked for in mid-stage and at the end, is the same in both, bit for bit."""
import numpy as np
import pytest
import torch

import helpers
from first_repo_gb300 import gen, pstep

pytestmark = pytest.mark.gpu


# (host fields are copied when they are bound: writing to them changes nothing)
@pytest.mark.parametrize("change,on_device", [
    ("bound", False), ("bound", True), ("bound_after_read", False), ("bound_after_read", True), ("written", True),
    ("coefficient", False), ("coefficient", True)])
def test_what_the_advance_saw(built_cuda, change, on_device):
    n, count = 12, 1500
    bp = helpers.make_bp(n, count)
    case = gen.make_case(n, count, 4, True)
    arrs = [np.ascontiguousarray(case[k]) for k in ("x", "y", "z", "u", "v", "w", "t", "flag")]
    fields = helpers.ghosted_fields(case)
    first, second = fields[3], gen.ghost(gen.make_case(n, 8, 17, False)["T"] + 0.3)

    def put(a):
        return torch.from_numpy(a).cuda() if on_device else a

    def run(late):
        g = pstep.ParticleStep(bp.step_config(), count, pstep.FP64, pstep.TRACK_ORDER)
        g.load(*arrs)
        g.bind_velocity(*fields[:3])
        bound = put(first.copy())
        g.bind_temperature(bound)
        g.prime()
        for k in range(4):
            g.interp_advance_deposit(k)
            g.wrap()
            if late:
                g.bind_temperature(bound)
            g.stage_temp()
            g.end_stage()
        g.end_step()
        g.interp_advance_deposit(0)
        seen = []
        if change == "bound_after_read":
            seen.append(g.array("RHS_T"))
        if change in ("bound", "bound_after_read"):
            other = put(second)
            g.bind_temperature(other)
        elif change == "written":
            torch.cuda.synchronize()
            bound.copy_(put(second))
            torch.cuda.synchronize()
        else:
            c = pstep.make_config(dict(bp.step_config(), nu=1.7 * bp.step_config()["nu"]), count, pstep.FP64,
                                  pstep.TRACK_ORDER)
            g._ok(g.L.pstep_update_params(g.h, c))
        seen.append(g.array("RHS_T"))
        g.wrap()
        seen.append(g.array("RHS_T"))
        g.stage_temp()
        seen += [g.array("RHS_T"), g.field("RHS_Part_Temp")]
        g.end_stage()
        g.stage(1)
        seen += [g.array("T_new"), g.array("RHS_T")]
        assert g.check() == (0, 0)
        g.close()
        return seen

    for a, b in zip(run(True), run(False), strict=True):
        assert helpers.bits_equal(a, b)
