"""The one-pass scan of the voxel counts at the edges of its tiles (4096
entries) and of its look-back window (32 tiles)."""
import numpy as np
import pytest

from gpu_util import to_device, torch_cuda

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(1, 1, 1), (15, 13, 21), (16, 16, 16), (31, 33, 8), (64, 64, 32),
                                  (51, 52, 50), (128, 128, 80)])
@pytest.mark.parametrize("n", [1, 5000])
def test_table_is_the_prefix_of_the_counts(dims, n):
    torch_cuda()
    from sphgb import kernels as K
    from sphgb.device import SceneBatch
    from test_gpu_density_paths import _fill, _spec
    space = tuple(0.125 * d for d in dims)
    pos, vel = _fill(n, space, seed=n + sum(dims))
    b = SceneBatch([_spec(n, space, 0.125, 32)])
    assert b.n_voxels == dims[0] * dims[1] * dims[2] + 1      # and the overflow entry
    p4, v4, pid, _ = to_device(pos, vel)
    for _ in range(3):                                        # the status words start over
        _, _, ids, _, start, count = K.organize_voxels(b, p4, v4, pid)
        c = count.cpu().numpy()
        vox = K.assign_voxels_to_particles(b, p4).cpu().numpy()
        np.testing.assert_array_equal(c, np.bincount(vox, minlength=b.n_voxels))
        np.testing.assert_array_equal(start.cpu().numpy(), np.concatenate([[0], np.cumsum(c)[:-1]]))
        np.testing.assert_array_equal(ids.cpu().numpy(), np.argsort(vox, kind="stable"))
    b.close()
