"""The FP32 deposit without tiles (a particle in eight cells or fewer, from 128^3 cells on): a word per cell and
field with the tiles' handling of overflows. The sums are integers, so it has to agree exactly with the
deposit by tiles: a population that is thin gives, taken twice over, which is not, exactly twice the
fields. Cells whose sums pass 2^31, bricks past a work item's size (8192), fast movers, positions on the
faces of bricks and of the box, an odd grid; against the oracle as tests/test_deposit_tiles_gpu.py does; and
handles on which thin and crowded populations take turns, with momentum and without, against fresh ones."""
import numpy as np
import pytest

import helpers
import pyoracle
from first_repo_gb300 import gen, pstep
from test_deposit_tiles_gpu import outputs, population, start

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,count,per_cell,speed", [
    (128, 140000, 600, 0.2), (128, 140000, 8300, 0.9), (136, 160000, 2000, 0.1)])
def test_thin_and_tiled_agree(built_cuda, n, count, per_cell, speed):
    bp, arrs = population(n, count, per_cell, 5, speed)
    dx = bp.l / n
    edge = np.random.default_rng(1).integers(0, 2 * n, (3, 3000)) * (0.5 * dx)  # cell and brick faces, half cells
    for d in range(3):
        arrs[d][-3000:] = np.minimum(edge[d], np.nextafter(bp.l, 0.0))
    fields = helpers.ghosted_fields(gen.make_case(n, 8, 5, False))
    assert 8 * count <= n ** 3 < 16 * count
    once = start(pstep.ParticleStep(bp.step_config(), count, pstep.FP32, 0), arrs, fields)
    primed = once.field("RHS_Part_Temp")
    once.run(2)
    a = outputs(once)
    twice = start(pstep.ParticleStep(bp.step_config(), 2 * count, pstep.FP32, 0),
                  [np.concatenate([q, q]) for q in arrs], fields)
    assert helpers.bits_equal(twice.field("RHS_Part_Temp"), 2.0 * primed)
    twice.run(2)
    b = outputs(twice)
    for k in a:
        assert helpers.bits_equal(b[k], 2.0 * a[k]), k
    assert once.check() == twice.check() == (0, 0)


def test_thin_against_the_oracle(built_cuda):
    n, count = 128, 3000
    bp, arrs = population(n, count, 200, 9, 0.3)
    fields = helpers.ghosted_fields(gen.make_case(n, 8, 5, False))
    o = pyoracle.Oracle(bp.step_config(), count)
    o.load(*arrs, np.arange(count, dtype=np.int32))
    o.prime(fields[3])
    o.run(1, *fields)
    g = start(pstep.ParticleStep(bp.step_config(), count, pstep.FP32, 0), arrs, fields)
    g.run(1)
    a = outputs(g)
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
    assert g.check() == (0, 0)


def test_thin_and_crowded_in_turn(built_cuda):
    n, cap = 128, 300000
    bp, many = population(n, cap, 9000, 7, 0.2)
    _, some = population(n, 200000, 300, 8, 0.2)
    _, few = population(n, 9, 3, 10, 0.2)
    fields = helpers.ghosted_fields(gen.make_case(n, 8, 5, False))
    nobody = [q[:0] for q in few]

    def config(on):
        return dict(bp.step_config(), twc=on)

    g = pstep.ParticleStep(config(1), cap, pstep.FP32, 0)
    g.load(*few, np.arange(9, dtype=np.int32))  # the same reference temperature everywhere
    for at, (arrs, on, steps) in enumerate(((many, 1, 1), (some, 1, 2), (many, 0, 1), (few, 0, 1), (some, 1, 0), (many, 1, 1),
                                            (nobody, 1, 1), (many, 0, 1), (some, 0, 1), (many, 1, 2), (few, 1, 1))):
        g._ok(g.L.pstep_update_params(g.h, pstep.make_config(config(on), cap, pstep.FP32, 0)))
        f = pstep.ParticleStep(config(on), cap, pstep.FP32, 0)
        f.load(*few, np.arange(9, dtype=np.int32))
        for h in (g, f):
            start(h, arrs, fields)
        assert helpers.bits_equal(g.field("RHS_Part_Temp"), f.field("RHS_Part_Temp")), at
        if steps:
            g.run(steps)
            f.run(steps)
            a, b = outputs(g), outputs(f)
            for k in a:
                assert helpers.bits_equal(a[k], b[k]), (at, k)
        f.close()
    assert g.check() == (0, 0)
    g.close()
