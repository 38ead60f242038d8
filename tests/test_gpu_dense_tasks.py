"""Tasks of dense voxels, which contexts of the tensor-core density pass hand to
the ballot pass: dense scenes beside sparse and uncapped ones, and dense
clusters in large sparse tables, on both sides of the voxel size where the
lists part.  Against the thread-per-particle pass, bit for bit."""
import numpy as np
import pytest

from gpu_util import torch_cuda

pytestmark = pytest.mark.gpu


def _scene(n, space, cap, seed, fill=None, at=0.0):
    from test_gpu_density_paths import _fill, _spec
    pos, vel = _fill(n, (fill or space,) * 3, seed)
    return _spec(n, (space,) * 3, 0.1, cap, mass=4.0 / n), pos + np.float32(at), vel


@pytest.mark.parametrize("per_voxel", [40, 63, 66, 133, 200])
@pytest.mark.parametrize("beside", [[(2000, 0.8, 0)], [(2000, 0.8, 32)], [(6000, 0.4, 0), (900, 0.8, 7)],
                                    [(3000, 0.8, 40), (2000, 0.8, 32)]])
def test_dense_scene_beside_others(per_voxel, beside):
    torch_cuda()
    from test_gpu_density_paths import _both
    parts = [_scene(per_voxel * 216, 0.6, 32, seed=per_voxel)]
    parts += [_scene(n, space, cap, seed=k) for k, (n, space, cap) in enumerate(beside)]
    for order in (parts, parts[::-1]):
        _both([p[0] for p in order], [p[1] for p in order], [p[2] for p in order])


@pytest.mark.parametrize("n", [262_144, 262_145, 300_000])
@pytest.mark.parametrize("cap", [32, 5])
def test_cluster_in_a_large_sparse_scene(n, cap):
    """Half of the particles at a few per voxel, half in a cluster of 150 to 250."""
    torch_cuda()
    from test_gpu_density_paths import _both, _spec
    rng = np.random.default_rng(n + cap)
    pos = (rng.random((n, 3)) * 5.0).astype(np.float32)
    k = n // 2
    pos[:k] = (1.0 + 0.87 * rng.random((k, 3))).astype(np.float32)
    ids = rng.permutation(n)
    pos = pos[ids].astype(np.float64)
    vel = (rng.standard_normal((n, 3)) * 0.1).astype(np.float32).astype(np.float64)
    _both([_spec(n, (5.0, 5.0, 5.0), 0.1, cap, mass=1e-4)], [pos], [vel])
