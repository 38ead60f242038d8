"""Steps in one call (each clears the counts of the one after it) against as
many calls of one step: odd and even numbers, graphs and plain launches, small
tables and one beyond the size that has two count buffers.  Compared in original
order: particles that went non-finite have no defined place in the slot order."""
import numpy as np
import pytest

from gpu_util import torch_cuda

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,h,mass", [(1, 0.1, 0.008), (3000, 0.1, 0.008), (20_000, 0.1, 0.008),
                                      (4000, 0.009, 0.008), (4000, 0.009, 1e-7), (4000, 0.0075, 1e-7)])
@pytest.mark.parametrize("cap", [32, 0])
def test_steps_in_one_call(n, h, mass, cap):
    torch_cuda()
    from sphgb.data_classes import SimulationState
    from sphgb.device import SceneBatch
    from test_gpu_density_paths import _fill, _spec
    pos, vel = _fill(n, (1.0, 1.0, 1.0), seed=n)
    spec = _spec(n, (1.0, 1.0, 1.0), h, cap, mass=mass)

    def run(calls, use_graph):
        b = SceneBatch([spec])
        b.load_states([SimulationState(pos, vel, np.zeros(n))])
        for k in calls:
            b.step(k, use_graph=use_graph)
        out = [t.cpu().numpy().copy() for t in (b.pos, b.vel, b.rho, b.pid, *b.step_neighbours())]
        b.close()
        order = np.argsort(out[3])
        return [t[order] for t in out[:3]] + out[4:]

    want = run([1] * 9, False)
    for calls in ([9], [4, 5], [2, 1, 3, 3], [1, 2, 2, 4]):
        for use_graph in (False, True):
            for a, c in zip(run(calls, use_graph), want):
                np.testing.assert_array_equal(a, c, err_msg=str((calls, use_graph)))
