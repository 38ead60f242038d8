"""Density tasks of two voxels (tiled scenes of more particles than the first
warps take) against the thread-per-particle pass: rows, counts, densities and
the next state bit for bit, at the edges of what a pair may hold."""
import numpy as np
import pytest

from gpu_util import torch_cuda
from test_gpu_density_paths import _both, _fill, _spec

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("a,b", [(1, 1), (8, 8), (9, 8), (15, 1), (1, 15), (16, 1), (2, 15)])
@pytest.mark.parametrize("cap", [32, 5, 0])
def test_counts_of_the_two_voxels(a, b, cap):
    """a particles in each voxel of even z and b in each of odd z; the last
    layer (an odd number of them) has no partner."""
    torch_cuda()
    h, nz = 0.125, 11
    side = 34 if a + b == 2 else 14
    rng = np.random.default_rng(100 * a + b)
    cells = np.stack(np.meshgrid(np.arange(side), np.arange(side), np.arange(nz), indexing="ij"),
                     axis=-1).reshape(-1, 3)
    cells = np.repeat(cells, np.where(cells[:, 2] % 2 == 0, a, b), axis=0)
    cells = cells[rng.permutation(len(cells))]
    pos = ((cells + rng.random(cells.shape, dtype=np.float32) * 0.999) * h).astype(np.float32)
    vel = rng.standard_normal(pos.shape, dtype=np.float32) * np.float32(0.1)
    n = len(pos)
    assert n > 10_000
    _both([_spec(n, (side * h, side * h, nz * h), h, cap)], [pos.astype(np.float64)],
          [vel.astype(np.float64)])


@pytest.mark.parametrize("per_voxel", [0.7, 4.0, 8.0])
@pytest.mark.parametrize("voxel", [(0.1, 0.1, 0.1), (0.12, 0.1, 0.11), (0.1, 0.11, 0.09)])
@pytest.mark.parametrize("cap", [32, 0])
def test_occupancies_and_voxels(per_voxel, voxel, cap):
    """Pairs and single voxels mixed, odd table sizes, and voxels less deep than
    the radius (no pairs: the walk they leave out may hold neighbours)."""
    torch_cuda()
    nx, nz = (29, 27) if per_voxel < 1 else (15, 17)
    space = tuple(float(np.float32(k * v)) for k, v in zip((nx, nx, nz), voxel))
    n = max(int(per_voxel * nx * nx * nz), 10_500)
    pos, vel = _fill(n, space, seed=n)
    _both([_spec(n, space, 0.1, cap, voxel=voxel)], [pos], [vel])


@pytest.mark.parametrize("cap", [32, 0])
def test_lattice_at_the_radius(cap):
    """Columns of particles one radius apart in z, on the voxels' own edges and
    one unit in the last place on either side."""
    torch_cuda()
    h = np.float32(0.1)
    x = (np.arange(24) * 0.06 + 0.01).astype(np.float32)
    z = (np.arange(21) * h).astype(np.float32)
    z = np.concatenate([z, np.nextafter(z, np.float32(9)), np.nextafter(z, np.float32(0))])
    pos = np.stack(np.meshgrid(x, x, z, indexing="ij"), axis=-1).reshape(-1, 3).astype(np.float64)
    rng = np.random.default_rng(3)
    pos = pos[rng.permutation(len(pos))][:20_000]
    _both([_spec(len(pos), (1.5, 1.5, 2.1), 0.1, cap)], [pos], [np.zeros_like(pos)])


def test_several_scenes():
    """Tables of different sizes end to end, particles outside them and
    non-finite ones included."""
    torch_cuda()
    specs, poss, vels = [], [], []
    for i, (n, side) in enumerate([(1, 0.3), (900, 0.7), (9000, 1.1), (4000, 0.9), (37, 0.5)]):
        pos, vel = _fill(n, (side, side * 0.8, side * 1.3), seed=i)
        if n > 100:
            pos[3] = (side * 1.4, 0.1, 0.2)
            pos[5] = (0.1, 0.2, -0.3)
            pos[7, 2] = np.inf
        specs.append(_spec(n, (side, side * 0.8, side * 1.3), 0.1, 32))
        poss.append(pos)
        vels.append(vel)
    _both(specs, poss, vels)
