"""The counting rank of the voxel sort: runs of every length up to two loads of
eight ids and beyond, starting at every alignment, against a sort on the host."""
import numpy as np
import pytest

from gpu_util import to_device, torch_cuda

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("last", [1, 7, 8, 9, 17, 64])
@pytest.mark.parametrize("rows64", [False, True])
def test_runs(last, rows64):
    torch_cuda()
    from sphgb import kernels as K
    from sphgb.device import SceneBatch
    from test_gpu_density_paths import _spec
    side, h = 6, 0.25
    rng = np.random.default_rng(last)
    counts = rng.integers(0, last + 1, side ** 3)
    counts[0], counts[1], counts[-1] = last, 1, last
    ids = np.repeat(np.arange(side ** 3), counts)[rng.permutation(counts.sum())]
    n = len(ids)
    cells = np.stack([ids % side, ids // side % side, ids // side ** 2], axis=-1)
    pos = ((cells + rng.random((n, 3), dtype=np.float32) * 0.99) * h).astype(np.float32)
    vel = rng.random((n, 3), dtype=np.float32)
    b = SceneBatch([_spec(n, (side * h,) * 3, h, 32)])
    p4, v4, pid, p64 = to_device(pos.astype(np.float64), vel.astype(np.float64))
    out = K.organize_voxels(b, p4, v4, pid, p64 if rows64 else None)
    order = np.lexsort((np.arange(n), ids))
    np.testing.assert_array_equal(out[2].cpu().numpy(), order)
    np.testing.assert_array_equal(out[0].cpu().numpy()[:, :3], pos[order])
    np.testing.assert_array_equal(out[1].cpu().numpy()[:, :3], vel[order])
    if rows64:
        np.testing.assert_array_equal(out[3].cpu().numpy(), pos[order].astype(np.float64))
    np.testing.assert_array_equal(out[5].cpu().numpy()[:side ** 3], counts)
    b.close()
