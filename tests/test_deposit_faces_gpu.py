"""The FP64 brick deposit's face sums keep the accuracy of their terms: particles just below a cell's upper faces give
its lower faces (1 - x_l) r with 1 - x_l near 2^-20. Two of them in every other cell, all RHS_u of one
sign, against the reference's sums: there a term is rounded once (1 - x_l is exact) and two are added, here
a term is rounded once and two are added, so the two agree to 4 x 2^-53 of the value, at the lower faces
as at the upper ones. (As sum r - sum x_l r the lower faces keep 33 bits.)"""
import numpy as np
import pytest

import helpers
from first_repo_gb300 import gen, pstep

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("same_class", [True, False])
def test_small_face_terms_keep_their_digits(built_cuda, same_class):
    n = 12
    cells = np.stack(np.meshgrid(*[np.arange(0, n, 2)] * 3, indexing="ij")).reshape(3, -1)
    count = 2 * cells.shape[1]
    bp = helpers.make_bp(n, count)
    dx = bp.l / n
    near = np.repeat([[1.0 - 2.0 ** -20], [1.0 - 2.0 ** -21]], cells.shape[1], axis=1).reshape(-1)
    x = np.concatenate([cells, cells], axis=1) + near
    if not same_class:  # the second one of a cell in another half of it along x: another class, its x terms not small
        x[0, cells.shape[1]:] -= 0.6
    vel = np.full((3, count), -5.0)  # slower than the gas everywhere: RHS_u > 0
    arrs = [np.ascontiguousarray(a) for a in (*(x * dx), *vel, np.ones(count))]
    fields = helpers.ghosted_fields(gen.make_case(n, 8, 5, False))
    got = []
    for flags in (pstep.TRACK_ORDER, pstep.TRACK_ORDER | pstep.REFERENCE_SUMS):
        g = pstep.ParticleStep(bp.step_config(), count, pstep.FP64, flags)
        g.load(*arrs, np.arange(count, dtype=np.int32))
        g.bind_velocity(*fields[:3])
        g.bind_temperature(fields[3])
        g.prime()
        g.interp_advance_deposit(0)
        got.append([g.field(k)[1:-1, 1:-1, 1:-1] for k in ("RHS_RU_x", "RHS_RU_y", "RHS_RU_z")])
        g.close()
    for d, (a, b) in enumerate(zip(*got, strict=True)):
        if d or same_class:
            assert 0.0 < b[b > 0].min() < 1e-5 * b.max()
        assert np.all((a > 0) == (b > 0))
        assert np.all(np.abs(a - b) <= 4 * 2.0 ** -53 * b), float(np.max(np.abs(a - b)[b > 0] / b[b > 0]))
