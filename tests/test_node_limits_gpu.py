"""The FP64 form's lists a node around the lengths where their handling changes or has changed: 31 to 34 and 63 to
66 particles a node (one thread's, or a warp's in the brick deposit) and 16383 to 16385 (16384 is the longest list sorted on
chip; one more is reported as PSTEP_ERR_CAPACITY, in bounds, and the handle goes on). Fields by bricks
against the reference's sums within the form's 1e-12 of max|field| (tests/test_deposit_lists_gpu.py);
the reference's sums and order against the oracle, bit for bit."""
import numpy as np
import pytest

import helpers
import pyoracle
from first_repo_gb300 import gen, pstep

pytestmark = pytest.mark.gpu


def crowd(n, per_node, rest, seed):
    count = 2 * per_node + rest
    bp = helpers.make_bp(n, count)
    dx = bp.l / n
    rng = np.random.default_rng(seed)
    x = rng.uniform(0.0, bp.l, (3, count))
    for at, node in enumerate((3.0, n - 2.0)):  # two full nodes, every h class
        x[:, at * per_node:(at + 1) * per_node] = (rng.uniform(-0.45, 0.45, (3, per_node)) + node) * dx
    x = x[:, rng.permutation(count)]
    vel = 0.02 * rng.normal(size=(3, count))
    arrs = [np.ascontiguousarray(a) for a in (*x, *vel, 1.0 + 0.1 * rng.normal(size=count))]
    return bp, arrs + [np.arange(count, dtype=np.int32)]


def start(g, arrs, fields):
    g.load(*arrs)
    g.bind_velocity(*fields[:3])
    g.bind_temperature(fields[3])
    g.prime()
    return g


@pytest.mark.parametrize("per_node", [31, 32, 33, 34, 63, 64, 65, 66])
def test_brick_lists_at_their_line(built_cuda, per_node):
    n = 13
    bp, arrs = crowd(n, per_node, 40, per_node)
    fields = helpers.ghosted_fields(gen.make_case(n, 8, 3, False))
    got = []
    for flags in (pstep.TRACK_ORDER, pstep.TRACK_ORDER | pstep.REFERENCE_SUMS):
        g = start(pstep.ParticleStep(bp.step_config(), len(arrs[0]), pstep.FP64, flags), arrs, fields)
        primed = g.field("RHS_Part_Temp")
        g.run(1)
        got.append([primed] + [g.field(k) for k in pstep.FIELD_IDS])
        assert g.check() == (0, 0)
        g.close()
    for a, b in zip(*got, strict=True):
        assert helpers.max_rel_to_max(a, b) <= 1e-12


@pytest.mark.parametrize("per_node", [16383, 16384])
def test_longest_sorted_lists_equal_the_oracle(built_cuda, per_node):
    n = 8
    bp, arrs = crowd(n, per_node, 37, per_node)
    fields = helpers.ghosted_fields(gen.make_case(n, 8, 5, False))
    o = pyoracle.Oracle(bp.step_config(), len(arrs[0]))
    o.load(*arrs)
    o.prime(fields[3])
    g = start(pstep.ParticleStep(bp.step_config(), len(arrs[0]), pstep.FP64, pstep.TRACK_ORDER | pstep.REFERENCE_SUMS),
              arrs, fields)
    assert g.check() == (0, 0)
    assert helpers.bits_equal(g.field("RHS_Part_Temp"), o.fields["E"])
    o.stage(0, *fields)
    g.stage(0)
    g.check()  # (a stage may gather a particle more at a node)
    assert helpers.bits_equal(g.array("flag"), o.flag())
    assert helpers.bits_equal(g.field("C"), o.fields["C"])
    g.close()


@pytest.mark.parametrize("flags", [pstep.TRACK_ORDER, pstep.TRACK_ORDER | pstep.REFERENCE_SUMS])
def test_one_particle_too_many_is_reported(built_cuda, flags):
    n = 8
    bp, arrs = crowd(n, 16385, 37, 5)
    few_bp, few = crowd(n, 60, 37, 6)
    fields = helpers.ghosted_fields(gen.make_case(n, 8, 5, False))
    g = start(pstep.ParticleStep(bp.step_config(), len(arrs[0]), pstep.FP64, flags), arrs, fields)
    assert g.check() == (3, 1 << 4)
    f = pstep.ParticleStep(bp.step_config(), len(arrs[0]), pstep.FP64, flags)
    for h in (g, f):
        start(h, few, fields)
        h.run(1)
        assert h.check() == (0, 0)
    for k in pstep.FIELD_IDS:
        assert helpers.bits_equal(g.field(k), f.field(k)), k
    for k in ("flag", "x", "T", "RHS_T"):
        assert helpers.bits_equal(g.array(k), f.array(k)), k
    g.close()
    f.close()
