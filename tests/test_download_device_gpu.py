"""pstep_download_particles into device arrays, FP64 form in the reference's order: exactly what
pstep_get_particle_array gives, between steps and within one, in arrays of their own and in ones that are not
aligned to their element; nothing beyond the particles is written."""
import ctypes as C

import numpy as np
import pytest
import torch

import helpers
from first_repo_gb300 import gen, pstep

pytestmark = pytest.mark.gpu

NAMES = ("x", "y", "z", "u", "v", "w", "T", "flag")


@pytest.mark.parametrize("count", [1, 257, 5000])
@pytest.mark.parametrize("shift", [0, 4])
def test_device_arrays(built_cuda, count, shift):
    n, spare = 12, 64
    bp = helpers.make_bp(n, count)
    case = gen.make_case(n, count, 4, True)
    g = pstep.ParticleStep(bp.step_config(), count + 10, pstep.FP64, pstep.TRACK_ORDER)
    g.load(*[np.ascontiguousarray(case[k]) for k in ("x", "y", "z", "u", "v", "w", "t", "flag")])
    fields = helpers.ghosted_fields(case)
    g.bind_velocity(*fields[:3])
    g.bind_temperature(fields[3])

    def check():
        size = [8 * count] * 7 + [4 * count]
        raw = [torch.full((s + spare,), 0x5A, dtype=torch.uint8, device="cuda") for s in size]
        torch.cuda.synchronize()
        at = [C.c_void_p(r.data_ptr() + shift) for r in raw]
        g._ok(g.L.pstep_download_particles(g.h, *at, 1))
        torch.cuda.synchronize()
        for name, r, s in zip(NAMES, raw, size, strict=True):
            b = r.cpu().numpy()
            assert b[shift:shift + s].tobytes() == np.ascontiguousarray(g.array(name)).tobytes(), name
            assert np.all(b[:shift] == 0x5A) and np.all(b[shift + s:] == 0x5A), name

    check()
    g.prime()
    check()
    g.run(3)
    check()
    g.stage(0)
    check()
    g.end_stage()
    check()
    g.close()
