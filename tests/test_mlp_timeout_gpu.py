"""A tensor-core completion wait that runs out in training (a barrier that nothing signals, polled by one
step's first wait under a short limit; the kernel drains its own MMA and frees its tensor memory): the
call reports it, the network is left as the step before left it, later calls change and write
nothing and report it too, and after the parameters are set again training goes on as on a fresh
handle, bit for bit. In a chunk that runs as a graph and in single steps, at the first step and later."""
import numpy as np
import pytest

from first_repo_gb300 import mlp

pytestmark = pytest.mark.gpu


def data():
    rng = np.random.default_rng(3)
    return rng.uniform(-1, 1, (4096, mlp.N_IN)).astype(np.float32), rng.normal(0, 0.5, (4096, mlp.N_OUT)).astype(np.float32)


@pytest.mark.parametrize("before,at,steps", [(0, 0, 3), (0, 2, 7), (5, 9, 60), (60, 0, 50), (3, 55, 120)])
def test_training_that_times_out(built_cuda, before, at, steps):
    x, y = data()
    net, ref = mlp.Mlp(seed=7), mlp.Mlp(seed=7)
    start = net.params
    for q in (net, ref):
        q.set_data(x, y)
        if before:
            q.train(before, batch=1024, seed=1)
    net.set_wait_limit(1000, before + at)
    with pytest.raises(mlp.MlpError, match="status 10"):
        net.train(steps, batch=1024, seed=2)
    # the steps before it, and nothing after
    if at:
        ref.train(at, batch=1024, seed=2)
    assert net.steps == ref.steps == before + at
    assert net.params.tobytes() == ref.params.tobytes()
    net.set_wait_limit()
    for call in (lambda: net.train(steps, batch=1024, seed=2), lambda: net.train(1, batch=1024, seed=2),
                 lambda: net.gradient(1024)):
        with pytest.raises(mlp.MlpError, match="status 10"):
            call()
        assert net.steps == before + at and net.params.tobytes() == ref.params.tobytes()
    # the parameters set again: as a fresh handle (no tensor memory was left allocated)
    for q in (net, ref):
        q.params = start
    a, b = net.train(steps, batch=1024, seed=4), ref.train(steps, batch=1024, seed=4)
    assert a.tobytes() == b.tobytes() and net.params.tobytes() == ref.params.tobytes() and net.steps == steps
    net.close()
    ref.close()


def test_gradient_that_times_out(built_cuda):
    x, y = data()
    net = mlp.Mlp(seed=7)
    net.set_data(x, y)
    before, _ = net.gradient(1024)
    start = net.params
    net.set_wait_limit(1000, 0)
    with pytest.raises(mlp.MlpError, match="status 10"):
        net.gradient(1024)
    net.set_wait_limit()
    net.params = start
    assert net.gradient(1024)[0].tobytes() == before.tobytes()
    net.close()
