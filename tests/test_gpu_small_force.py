"""The force pass of small contexts (eight lanes per particle) against the one
of large contexts (a thread per particle): a scene gives the same bits alone and
beside scenes that take its context over the limit."""
import numpy as np
import pytest

from gpu_util import torch_cuda

pytestmark = pytest.mark.gpu


def _state(b, k, n):
    pos, vel, rho = (t.cpu().numpy() for t in b.export_aos_f64())
    off = b.scene_offsets[k]
    return pos[off:off + n], vel[off:off + n], rho[off:off + n]


@pytest.mark.parametrize("n", [1, 2, 7, 31, 33, 257, 4000])
@pytest.mark.parametrize("cap,spread", [(32, 0.35), (5, 0.35), (0, 0.35), (32, 1.0)])
def test_alone_and_beside_a_large_scene(n, cap, spread):
    """spread 1.0: few neighbours, densities of 0 and non-finite factors (the
    deferred particles); cap 0: rows that do not hold every neighbour."""
    torch_cuda()
    from sphgb.data_classes import SimulationState
    from sphgb.device import SceneBatch
    from test_gpu_density_paths import _fill, _spec
    pos, vel = _fill(n, (spread,) * 3, seed=n + cap)
    spec = _spec(n, (1.0, 1.0, 1.0), 0.1, cap)
    big_pos, big_vel = _fill(30_000, (1.0, 1.0, 1.0), seed=2)
    big = _spec(30_000, (1.0, 1.0, 1.0), 0.1, 32)
    one, two = SceneBatch([spec]), SceneBatch([spec, big])
    small = SimulationState(pos, vel, np.zeros(n))
    one.load_states([small])
    two.load_states([small, SimulationState(big_pos, big_vel, np.zeros(30_000))])
    one.step(2)
    two.step(2)
    for a, c in zip(_state(one, 0, n), _state(two, 0, n)):
        np.testing.assert_array_equal(a, c)
    # a frozen scene keeps its state through the pass
    one.set_step_limits([2])
    before = _state(one, 0, n)
    one.step(1)
    for a, c in zip(before, _state(one, 0, n)):
        np.testing.assert_array_equal(a, c)
    one.close()
    two.close()
