"""The FP32 deposit's tiles and 64-bit sums where their handling changes: bricks at and past the size of
one work item (8192 particles), cells whose sums pass 2^31, positions more than half a cell outside
their brick, neighbours that wrap onto each other (two bricks a side), partial rows of 32 cells, and
populations that leave tiles behind. The sums are integers, so what has to hold holds exactly:
a population uploaded twice over deposits exactly twice the fields, and a used handle gives what
a fresh one gives. Against the oracle: the form's 1e-5 of max|field|; the momentum deposit is
piecewise constant across the axes, so a particle within fp32 resolution of a cell face may deposit
in the neighbouring cell (fast movers meet one now and then): such cells are few, and the difference
cancels in the sum."""
import numpy as np
import pytest

import helpers
import pyoracle
from first_repo_gb300 import gen, pstep

pytestmark = pytest.mark.gpu


def population(n, count, per_cell, seed, speed):
    bp = helpers.make_bp(n, count)
    rng = np.random.default_rng(seed)
    dx = bp.l / n
    x = rng.uniform(0.0, bp.l, (3, count))
    crowd = min(per_cell, count)
    x[:, :crowd] = (np.array([[n - 1.0], [7.0], [8.0]]) + rng.uniform(0.0, 1.0, (3, crowd))) * dx
    v = rng.uniform(-1.0, 1.0, (3, count)) * speed * dx / bp.dt  # cells per step
    t = 1.0 + 0.1 * rng.normal(size=count)
    return bp, [np.ascontiguousarray(a) for a in (*x, *v, t)]


def start(g, arrs, fields):
    g.load(*arrs, np.arange(len(arrs[0]), dtype=np.int32))
    g.bind_velocity(*fields[:3])
    g.bind_temperature(fields[3])
    g.prime()
    return g


def outputs(g):
    return {**{k: g.field(k) for k in pstep.FIELD_IDS}, "mom": g.momentum_sums(), "mean": np.array(g.energy_mean()),
            "stats": np.array([g.field_stats(k) for k in pstep.FIELD_IDS])}


@pytest.mark.parametrize("n,count,per_cell,speed", [
    (16, 2000, 300, 0.1), (24, 9000, 8192, 0.2), (40, 12000, 8193, 0.1), (72, 30000, 600, 0.3), (16, 3000, 50, 0.9),
    (40, 4000, 2, 0.9)])
def test_fields_against_the_oracle_and_doubling(built_cuda, n, count, per_cell, speed):
    bp, arrs = population(n, count, per_cell, 5, speed)
    fields = helpers.ghosted_fields(gen.make_case(n, 8, 5, False))
    o = pyoracle.Oracle(bp.step_config(), count)
    o.load(*arrs, np.arange(count, dtype=np.int32))
    o.prime(fields[3])
    o.run(1, *fields)
    once = start(pstep.ParticleStep(bp.step_config(), count, pstep.FP32, 0), arrs, fields)
    primed = once.field("RHS_Part_Temp")
    once.run(1)
    assert once.check() == (0, 0)
    a = outputs(once)
    for ours, theirs in (("C", "C"), ("RHS_RU_x", "Ax"), ("RHS_RU_y", "Ay"), ("RHS_RU_z", "Az"), ("RHS_Part_Temp", "E")):
        got, want = a[ours][1:-1, 1:-1, 1:-1], o.fields[theirs][1:-1, 1:-1, 1:-1]
        off, top = got - want, np.abs(want).max()
        if ours.startswith("RHS_RU"):
            assert np.count_nonzero(np.abs(off) > 1e-5 * top) <= 8
            assert abs(off.sum()) <= 1e-5 * np.abs(want).sum(), ours
        else:
            assert np.abs(off).max() <= 1e-5 * top, ours
        assert helpers.bits_equal(a[ours][:, :, 0], a[ours][:, :, -2]) and helpers.bits_equal(a[ours][-1], a[ours][1])
        assert a["stats"][list(pstep.FIELD_IDS).index(ours)][0] == got.max()
        assert a["stats"][list(pstep.FIELD_IDS).index(ours)][1] == got.min()
    twice = start(pstep.ParticleStep(bp.step_config(), 2 * count, pstep.FP32, 0),
                  [np.concatenate([q, q]) for q in arrs], fields)
    assert helpers.bits_equal(twice.field("RHS_Part_Temp"), 2.0 * primed)
    twice.run(1)
    b = outputs(twice)
    for k in a:
        assert helpers.bits_equal(b[k], 2.0 * a[k]), k


def test_what_a_population_leaves_behind(built_cuda):
    n = 32
    bp, crowd = population(n, 9000, 8500, 7, 0.2)
    _, few = population(n, 40, 10, 8, 0.2)
    fields = helpers.ghosted_fields(gen.make_case(n, 8, 5, False))
    off = dict(bp.step_config(), twc=0)

    def fresh(arrs, cfg):
        g = pstep.ParticleStep(cfg, 9000, pstep.FP32, 0)
        g.load(*crowd, np.arange(len(crowd[0]), dtype=np.int32))  # the same reference temperature
        start(g, arrs, fields)
        primed = g.field("RHS_Part_Temp")
        g.run(1)
        return primed, outputs(g)

    g = pstep.ParticleStep(bp.step_config(), 9000, pstep.FP32, 0)
    twc = 1
    # momentum on and off, a prime without a step, crowds, a handful and nobody, in turn
    for arrs, on, steps in ((crowd, 1, 1), (few, 0, 1), (few, 1, 0), (crowd, 1, 0), (few, 1, 1), (crowd, 0, 1),
                            ([q[:0] for q in few], 1, 1), (few, 1, 1)):
        if on != twc:
            c = pstep.make_config(dict(bp.step_config(), twc=on), 9000, pstep.FP32, 0)
            g._ok(g.L.pstep_update_params(g.h, c))
            twc = on
        start(g, arrs, fields)
        primed, want = fresh(arrs, bp.step_config() if on else off)
        assert helpers.bits_equal(g.field("RHS_Part_Temp"), primed)
        if steps:
            g.run(1)
            got = outputs(g)
            for k in want:
                assert helpers.bits_equal(got[k], want[k]), k
