"""What a handle takes of the device's memory, against the bytes a particle and a cell that the forms are meant to
take, so that a population that fits a device goes on fitting: FP64 form in the reference's order 369 B a
particle and 60 B a cell, with the reference's sums no more (their order within a node lies in the order
passes' scratch); FP32 form 148 B a particle and 150 B a cell. Beside these, the device hands memory out in
pieces of 2 MB: at most one a array."""
import pytest
import torch

import helpers
from first_repo_gb300 import pstep

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,cap,precision,flags,per_particle,per_cell", [
    (64, 60_000_000, pstep.FP64, pstep.TRACK_ORDER, 369, 60),
    (64, 60_000_000, pstep.FP64, pstep.TRACK_ORDER | pstep.REFERENCE_SUMS, 369, 60),
    (64, 100_000_000, pstep.FP32, 0, 148, 150), (256, 1_000_000, pstep.FP32, 0, 148, 150),
    (256, 1_000_000, pstep.FP64, 0, 369, 60)])
def test_memory_of_a_handle(built_cuda, n, cap, precision, flags, per_particle, per_cell):
    bp = helpers.make_bp(n, cap)
    pstep.ParticleStep(bp.step_config(), 16, precision, flags).close()  # the library's own
    torch.cuda.synchronize()
    free, _ = torch.cuda.mem_get_info()
    g = pstep.ParticleStep(bp.step_config(), cap, precision, flags)
    taken = free - torch.cuda.mem_get_info()[0]
    g.close()
    assert taken <= per_particle * cap + per_cell * (n + 2) ** 3 + 100 * (2 << 20), taken
    assert torch.cuda.mem_get_info()[0] >= free - (2 << 20)
