"""The counting sort's ways of adding for several particles at once: populations in one, a few, some tens and
many cells, uploaded in no order, in storage order, and shuffled within blocks of 64, give the same
integer sums in the FP32 form, bit for bit, and every particle comes back once."""
import numpy as np
import pytest

import helpers
from first_repo_gb300 import gen, pstep

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells", [1, 2, 5, 9, 40, 3000])
def test_order_of_upload_does_not_show(built_cuda, cells):
    n, count = 32, 20011
    bp = helpers.make_bp(n, count)
    rng = np.random.default_rng(cells)
    at = rng.integers(0, n, (3, cells))[:, rng.integers(0, cells, count)]
    x = (at + rng.uniform(0.0, 1.0, (3, count))) * (bp.l / n)
    arrs = [*x, *(0.1 * (bp.l / n / bp.dt) * rng.uniform(-1, 1, (3, count))), 1.0 + 0.1 * rng.normal(size=count)]
    arrs[6][:] = np.round(arrs[6] * 1024.0) / 1024.0  # exact offsets from any of them: the first one is the reference
    fields = helpers.ghosted_fields(gen.make_case(n, 8, 5, False))
    brick = (at[2] // 8 * (n // 8) + at[1] // 8) * (n // 8) + at[0] // 8
    by_cell = np.lexsort((at[0], at[1], at[2], brick))
    nearly = by_cell.copy()
    for b in range(0, count - 64, 64):
        nearly[b:b + 64] = rng.permutation(nearly[b:b + 64])
    want = None
    for order in (by_cell, rng.permutation(count), nearly):
        g = pstep.ParticleStep(bp.step_config(), count, pstep.FP32, 0)
        g.load(*[np.ascontiguousarray(a[:1]) for a in arrs], np.zeros(1, dtype=np.int32))  # the reference temperature
        g.load(*[np.ascontiguousarray(a[order]) for a in arrs], order.astype(np.int32))
        g.bind_velocity(*fields[:3])
        g.bind_temperature(fields[3])
        g.prime()
        g.run(2)
        ids = g.array("flag")
        assert np.array_equal(np.sort(ids), np.arange(count))
        got = [g.field(k) for k in pstep.FIELD_IDS] + [g.array(k)[np.argsort(ids)] for k in ("x", "u", "T")]
        want = want or got
        for a, b in zip(got, want, strict=True):
            assert helpers.bits_equal(a, b)
        assert g.check() == (0, 0)
        g.close()
