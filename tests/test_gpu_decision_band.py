"""Pairs whose squared distance is a few 1e-5 of the voxel side squared from the
radius squared: where the tensor-core decision of k_density_tc must hand over to
the exact one.  Against the thread-per-particle pass, bit for bit."""
import numpy as np
import pytest

from gpu_util import torch_cuda

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("per_voxel", [6, 11])
@pytest.mark.parametrize("cap", [32, 0])
@pytest.mark.parametrize("seed", [1, 2, 3])
def test_pairs_near_the_radius(per_voxel, cap, seed):
    """Every second particle lies at h (1 + e) from the one before it, |e| up to
    1.5e-4, on both sides: (d^2 - h^2) / side^2 up to 3e-4 around the tolerance
    of 1e-4."""
    torch_cuda()
    from test_gpu_density_paths import _both, _spec
    rng = np.random.default_rng(seed)
    h, half = 0.1, per_voxel * 500
    a = 0.15 + 0.7 * rng.random((half, 3))
    u = rng.standard_normal((half, 3))
    u /= np.linalg.norm(u, axis=1)[:, None]
    e = rng.uniform(-1.5e-4, 1.5e-4, (half, 1))
    a = a.astype(np.float32).astype(np.float64)
    b = (a + u * float(np.float32(h)) * (1.0 + e)).astype(np.float32).astype(np.float64)
    pos = np.stack([a, b], axis=1).reshape(-1, 3)
    d = np.linalg.norm(pos[0::2] - pos[1::2], axis=1) / float(np.float32(h)) - 1.0
    band = np.abs(2.0 * d)
    assert ((band > 4e-5) & (band < 1.2e-4)).sum() > half // 6       # the tolerance's surroundings
    pos = pos[rng.permutation(2 * half)]
    vel = rng.normal(0, 0.1, pos.shape).astype(np.float32).astype(np.float64)
    _both([_spec(2 * half, (1.0, 1.0, 1.0), h, cap, mass=1e-3)], [pos], [vel])
