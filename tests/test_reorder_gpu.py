"""The per-step reorder (all arrays in one launch, with and without a tau_p of each particle's own)
and the base state's download, together between steps and one array at a time within one: the
same values and ids as the single arrays and, in the reference's order, the oracle's, exactly."""
import numpy as np
import pytest

import helpers
import pyoracle
from first_repo_gb300 import gen, pstep

pytestmark = pytest.mark.gpu
NAMES = ["x", "y", "z", "u", "v", "w", "T", "flag"]


def download(g, count):
    out = [np.empty(count) for _ in range(7)] + [np.empty(count, dtype=np.int32)]
    g.download(*out)
    return out


@pytest.mark.parametrize("count", [1, 257, 5000])
@pytest.mark.parametrize("order", [0, pstep.TRACK_ORDER])
@pytest.mark.parametrize("tau", [False, True])
def test_reorder_and_download(built_cuda, count, order, tau):
    n = 10
    bp = helpers.make_bp(n, count)
    cfg = bp.step_config()
    case = gen.make_case(n, count, 7, True)
    arrays = [np.ascontiguousarray(case[k]) for k in ("x", "y", "z", "u", "v", "w", "t", "flag")]
    ux, uy, uz, tf = helpers.ghosted_fields(case)
    o = None if tau else pyoracle.Oracle(cfg, count)
    g = pstep.ParticleStep(cfg, count, pstep.FP64, order)
    g.load(*arrays)
    if tau:
        g.set_tau_p(np.linspace(0.05, 0.2, count))
    g.bind_velocity(ux, uy, uz)
    g.bind_temperature(tf)
    for a, b in zip(download(g, count), arrays):
        assert np.array_equal(a, b)
    g.prime()
    if o:
        o.load(*arrays)
        o.prime(tf)
    for s in range(2):
        for k in range(4):
            g.stage(k)
            if o:
                o.stage(k, ux, uy, uz, tf)
            for name, a in zip(NAMES, download(g, count)):
                assert np.array_equal(a, g.array(name)), (s, k, name)
            g.end_stage()
            if o:
                o.end_stage()
        g.end_step()
        if o:
            o.end_step()
        got = download(g, count)
        for name, a in zip(NAMES, got):
            assert np.array_equal(a, g.array(name)), (s, name)
        if o:
            by, ref = np.argsort(got[7]), np.argsort(o.flag())
            if order:
                assert np.array_equal(got[7], o.flag())
            for name, a in zip(NAMES[:7], got):
                assert helpers.bits_equal(a[by], o.array(name)[ref]), (s, name)
    g.close()
