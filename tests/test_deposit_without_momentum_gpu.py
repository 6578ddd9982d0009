"""FP32 form without two-way coupling: bricks that hold no particles any more leave the deposit's work
lists, as they do with it, and their momentum sums of before are not seen when it is switched on again.

The lists show in the time of a step: a population in one corner (a 64th of the box) on a handle whose
former population was everywhere, against a fresh handle, in turn. Writing every brick's tile of
zeros again takes 4 x 70 us of about 1.3 ms a step at 256^3; the bound is a tenth."""
import numpy as np
import pytest
import torch

import helpers
from first_repo_gb300 import gen, pstep

pytestmark = pytest.mark.gpu


def population(n, count, bp, part, seed):
    rng = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.rand((3, count), generator=rng, device="cuda", dtype=torch.float64) * bp.l * part
    v = (torch.rand((3, count), generator=rng, device="cuda", dtype=torch.float64) - 0.5) * 0.1 * bp.l / n / bp.dt
    t = 1.0 + 0.02 * torch.rand(count, generator=rng, device="cuda", dtype=torch.float64)
    return [a.contiguous() for a in (*x, *v, t)] + [torch.arange(count, dtype=torch.int32, device="cuda")]


def start(g, arrs, fields):
    g.load(*arrs)
    g.bind_velocity(*fields[:3])
    g.bind_temperature(fields[3])
    g.prime()


def best_ms(g):
    g.run(2)
    times = []
    for _ in range(4):
        g.run(3)
        times.append(g.last_run_ms() / 3)
    return min(times)


def test_emptied_bricks_cost_nothing(built_cuda):
    n, count = 256, (1 << 21) + 9
    bp = helpers.make_bp(n, count, {"twc": 0})
    fields = [torch.from_numpy(a).cuda() for a in helpers.ghosted_fields(gen.make_case(n, 8, 3, False))]
    corner = population(n, count, bp, 0.25, 1)
    used, fresh = (pstep.ParticleStep(bp.step_config(), count, pstep.FP32, 0) for _ in range(2))
    start(used, population(n, count, bp, 1.0, 2), fields)
    used.run(1)
    for g in (used, fresh):
        start(g, corner, fields)
    a, b = min(best_ms(used), best_ms(used)), min(best_ms(fresh), best_ms(fresh))
    assert a <= 1.1 * b, (a, b)
    used.close()
    fresh.close()


@pytest.mark.parametrize("order", [(1, 0, 1), (0, 1), (1, 0, 0, 1), (1, 1, 0, 1, 0, 1)])
def test_momentum_switched_on_again(built_cuda, order):
    n = 32
    populations = [(20000, 1.0), (6000, 0.25), (9000, 0.5), (20000, 1.0), (700, 1.0), (6000, 0.25)]
    bp = helpers.make_bp(n, 20000)
    case = gen.make_case(n, 8, 5, False)
    fields = helpers.ghosted_fields(case)

    def config(on):
        return dict(bp.step_config(), twc=on)

    g = pstep.ParticleStep(config(order[0]), 20000, pstep.FP32, 0)
    first = population(n, 100, bp, 1.0, 99)  # (the same reference temperature everywhere)
    g.load(*first)
    for at, on in enumerate(order):
        count, part = populations[at]
        arrs = population(n, count, bp, part, at)
        g._ok(g.L.pstep_update_params(g.h, pstep.make_config(config(on), 20000, pstep.FP32, 0)))
        start(g, arrs, fields)
        g.run(2)
        f = pstep.ParticleStep(config(on), 20000, pstep.FP32, 0)
        f.load(*first)
        start(f, arrs, fields)
        f.run(2)
        for k in pstep.FIELD_IDS:
            assert helpers.bits_equal(g.field(k), f.field(k)), (at, k)
        assert np.array_equal(g.momentum_sums(), f.momentum_sums())
        f.close()
    assert g.check() == (0, 0)
    g.close()
