"""RK4 steps replayed as a graph: two captures (y and ynew swap roles), step
sizes that change between replays, a step with diagnostics in between."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu_mod():
    from instaheat_gb300 import gpu
    return gpu


@pytest.mark.parametrize("n", [(16, 16, 16), (24, 18, 12), (64, 32, 32)])
@pytest.mark.parametrize("prec", [0, 1])
def test_rk4_replay_is_identical(gpu_mod, n, prec):
    """The same steps kernel by kernel: bit-identical states, equal counters."""
    runs = []
    for graphs in (True, False):
        ctx = gpu_mod.Context(n=n, precision=prec)
        ctx.graphs(graphs)
        ctx.ic(seed=3)
        states = []
        for i, dt in enumerate([5e-3, 5e-3, 5e-3, 2e-3, 4e-3, 5e-3, 1e-3, 1e-3]):
            ctx.rk4_step(dt, output=(i == 5))
            states.append(ctx.get_state())
        runs.append((states, ctx.t, ctx.calls_rhs, ctx.kernel_launches))
        ctx.close()
    for a, b in zip(runs[0][0], runs[1][0]):
        assert np.array_equal(a, b)
    assert runs[0][1:] == runs[1][1:]
