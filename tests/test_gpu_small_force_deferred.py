"""Particles that the eight-lane force pass of small contexts defers because
their list does not fit its row: scenes without a cap whose context has no pool
of long lists (the thread-per-particle density variant), against the
thread-per-particle force pass of a context above the small pass's limit."""
import numpy as np
import pytest

from gpu_util import torch_cuda

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 40, 257, 4000, 20_000, 20_001])
def test_deferred_particles(n):
    torch_cuda()
    from sphgb import _capi
    from sphgb.data_classes import SimulationState
    from sphgb.device import SceneBatch
    from test_gpu_density_paths import _fill, _spec
    side = 0.45 * max(n / 4000.0, 0.02) ** (1.0 / 3.0)      # about 45 per voxel
    pos, vel = _fill(n, (side,) * 3, seed=n)
    spec = _spec(n, (1.0, 1.0, 1.0), 0.1, 0, mass=1.0 / n)
    big_pos, big_vel = _fill(30_000, (1.0, 1.0, 1.0), seed=2)
    big = _spec(30_000, (1.0, 1.0, 1.0), 0.1, 32)
    got = []
    for others in ([], [(big, big_pos, big_vel)]):
        b = SceneBatch([spec] + [o[0] for o in others])
        b.set_tuning(density_variant=_capi.DENSITY_THREAD)
        b.load_states([SimulationState(p, v, np.zeros(len(p)))
                       for p, v in [(pos, vel)] + [o[1:] for o in others]])
        b.step(2)
        if n > 40:
            count = b.step_neighbours()[1][:n].cpu().numpy()
            assert (count == -1).any()              # some particles are deferred
        got.append([t.cpu().numpy()[:n] for t in b.export_aos_f64()])
        b.close()
    for a, c in zip(*got):
        np.testing.assert_array_equal(a, c)
