"""Neighbour lists beyond 32 entries, whose room in the pool is taken before
they are written: walks of one chunk of candidates, a batch more, and several
chunks (counted first), caps just above a row, and pools that run out.  The
step and the stage calls against the thread-per-particle walk, bit for bit."""
import numpy as np
import pytest

from gpu_util import to_device, torch_cuda

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cap", [33, 48, 0])
@pytest.mark.parametrize("per_voxel,side", [(11.9, 1.0), (13.0, 1.0), (14.5, 1.0), (20.0, 0.8),
                                            (45.0, 0.5), (133.0, 0.4)])
def test_step_and_stages_equal_walks(per_voxel, side, cap):
    torch = torch_cuda()
    from sphgb import kernels as K
    from sphgb.device import SceneBatch
    from test_gpu_density_paths import _both, _fill, _spec
    from test_gpu_stage_lists import _stages
    n = int(per_voxel * (side / 0.1) ** 3)
    pos, vel = _fill(n, (side,) * 3, seed=n + cap)
    # the dense block alone (row-major table) and in a large box (tiled)
    for space in (side, max(1.0, 3.1 * side)):
        spec = _spec(n, (space,) * 3, 0.1, cap, mass=8.0 / n)
        _both([spec], [pos], [vel])
        b = SceneBatch([spec])
        p4, v4, pid, _ = to_device(pos, vel)
        pS, vS, idS, _, start, count = K.organize_voxels(b, p4, v4, pid)
        steps = torch.zeros(1, dtype=torch.int32, device="cuda")
        with_lists = [t.clone() for t in _stages(b, pS, vS, idS, start, count, steps)]
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            walked = _stages(b, pS, vS, idS, start, count, steps)
        graph.replay()
        torch.cuda.synchronize()
        for a, c in zip(with_lists, walked):
            np.testing.assert_array_equal(a.cpu().numpy(), c.cpu().numpy())
        b.close()


@pytest.mark.parametrize("walk", ["ceil", "truncated"])
def test_one_dense_spot_takes_the_pool(walk):
    """8,000 particles at 4 per voxel and 2,500 in one spot: their lists want
    more than the whole pool, so that some go there and the rest walk."""
    torch_cuda()
    from test_gpu_density_paths import _both, _fill, _spec
    pos, vel = _fill(10_500, (0.95,) * 3, seed=4)
    spot = np.random.default_rng(5).permutation(10_500)[:2_500]
    pos[spot] = np.asarray(0.31 + 0.14 * pos[spot], dtype=np.float32).astype(np.float64)
    _both([_spec(10_500, (0.95,) * 3, 0.1, 0, walk, mass=1e-4)], [pos], [vel])
