"""The integer fp32 <-> fp64 conversions of the FP32 form against the host's own (IEEE, round to
nearest even): an uploaded velocity comes back as float32 holds it, bit for bit, over the edges of
the normal range, ties, zeros, subnormals and infinities; a position as its trunc cell and fp32
offset give it. The counts leave a remainder in every block."""
import numpy as np
import pytest

from first_repo_gb300 import config, pstep

pytestmark = pytest.mark.gpu


def edge_values(count, seed):
    rng = np.random.default_rng(seed)
    bits = rng.integers(0, 1 << 52, count, dtype=np.uint64)
    exp = rng.integers(1023 - 160, 1023 + 140, count).astype(np.uint64)
    v = ((rng.integers(0, 2, count).astype(np.uint64) << np.uint64(63)) | (exp << np.uint64(52)) | bits).view(np.float64)
    f = np.float32(rng.normal(size=count)).astype(np.float64)
    ulp = np.spacing(np.abs(f).astype(np.float32)).astype(np.float64)
    v[::3] = f[::3] + 0.5 * ulp[::3]  # ties between two float32 values
    big = float(np.finfo(np.float32).max)
    special = [0.0, -0.0, 2.0 ** -126, 2.0 ** -126 * (1 - 2.0 ** -25), 2.0 ** -149, 2.0 ** -151, big,
               big * (1 + 2.0 ** -26), big * (1 + 2.0 ** -24), 2.0 ** 127, 1.0, -1.0, 1 - 2.0 ** -25]
    v[:min(count, len(special))] = special[:min(count, len(special))]
    return v


@pytest.mark.parametrize("count", [1, 31, 257, 4099])
def test_round_trip_is_the_float32_value(built_cuda, count):
    n = 16
    bp = config.box_params(n, count)
    g = pstep.ParticleStep(bp.step_config(), count, pstep.FP32, 0)
    rng = np.random.default_rng(count)
    pos = rng.uniform(0.0, bp.l, (3, count))
    pos[:, 0] = 0.0
    vel = np.stack([edge_values(count, 5 + d) for d in range(3)])
    t = np.ones(count)
    t[1:] += rng.normal(size=count)[1:]
    g.load(*[np.ascontiguousarray(a) for a in (*pos, *vel, t)], np.arange(count, dtype=np.int32))
    with np.errstate(over="ignore"):
        for d, name in enumerate("uvw"):
            assert g.array(name).tobytes() == vel[d].astype(np.float32).astype(np.float64).tobytes()
    assert g.array("T").tobytes() == ((t - 1.0).astype(np.float32).astype(np.float64) + 1.0).tobytes()
    for d, name in enumerate("xyz"):
        xi = pos[d] * (1.0 / (bp.l / n))
        c = np.floor(xi)
        o = (xi - c).astype(np.float32)
        c, o = np.where(o >= 1.0, c + 1, c) % n, np.where(o >= 1.0, np.float32(0), o)
        want = (c + o.astype(np.float64)) * (bp.l / n)
        # the offset may come from the product unrounded: half a float32 spacing of an offset below 1
        assert np.max(np.abs(g.array(name) - want)) <= 2.0 ** -24 * bp.l / n
    all_out = [np.empty(count) for _ in range(7)] + [np.empty(count, dtype=np.int32)]
    g.download(*all_out)
    for a, name in zip(all_out, ("x", "y", "z", "u", "v", "w", "T")):
        assert a.tobytes() == g.array(name).tobytes()
    g.close()


@pytest.mark.parametrize("n, dx", [(16, 1.0), (256, 0.3), (104, 2.0 * np.pi / 104)])
def test_downloaded_positions_are_rounded_once_each(built_cuda, n, dx):
    """(cell + offset) dx with one rounding in the product, over the offsets' whole range: zero, below and at
    2^-19 (where the sum needs no rounding), random ones and the largest below 1."""
    rng = np.random.default_rng(n)
    edge = np.array([0.0, 2.0 ** -30, 2.0 ** -19 * (1 - 2.0 ** -24), 2.0 ** -19, 2.0 ** -18, 0.5, 1 - 2.0 ** -24])
    o = np.concatenate([edge, 2.0 ** rng.uniform(-21, 0, 500), rng.uniform(0, 1, 500)]).astype(np.float32)
    o = np.minimum(np.tile(o, 3), np.float32(1 - 2.0 ** -24))
    cell = np.repeat([0.0, 1.0, n - 1.0], len(o) // 3)
    count = len(o)
    length = dx * n
    g = pstep.ParticleStep(dict(config.box_params(n, count).step_config(), l=length), count, pstep.FP32, 0)
    x = (cell + o.astype(np.float64)) * dx
    zero = np.zeros(count)
    g.load(x, zero, zero, zero, zero, zero, zero + 1.0, np.arange(count, dtype=np.int32))
    # the cell and fp32 offset the upload made of it, by the host
    xi = x * (1.0 / (length / n))
    c = np.floor(xi)
    f = (xi - c).astype(np.float32)
    c, f = np.where(f >= 1.0, c + 1, c) % n, np.where(f >= 1.0, np.float32(0), f)
    assert g.array("x").tobytes() == ((c + f.astype(np.float64)) * (length / n)).tobytes()
    g.close()
