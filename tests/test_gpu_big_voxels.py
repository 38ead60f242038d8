"""Voxels above the big-voxel threshold: their ids are sorted by counting up to
512 members and by a sorting network beyond; the organised state is the
reference's (voxel, particle id) order whatever the input order."""
import numpy as np
import pytest

from gpu_util import to_device, torch_cuda

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(64, 65, 66), (255, 256, 257, 1, 0, 3), (511, 512, 513, 1023, 1024, 1025),
                                   (2048, 5, 2049, 70), (9000, 100, 8192, 1024, 77), (8193,), (16384, 16385), (40_000, 3, 1200),
                                   (100_000,),
                                   tuple([133] * 40 + [1500] + [200] * 30)])
def test_order_of_big_voxels(sizes):
    torch = torch_cuda()
    from sphgb import kernels as K
    from sphgb.device import SceneBatch
    from test_gpu_density_paths import _spec
    rng = np.random.default_rng(len(sizes))
    cells = rng.choice(1000, size=len(sizes), replace=False)
    vid = np.repeat(cells, sizes)
    n = len(vid)
    xyz = np.stack([vid % 10, vid // 10 % 10, vid // 100], axis=1)
    pos = ((xyz + 0.2 + 0.6 * rng.random((n, 3))) * 0.1).astype(np.float32)
    order = rng.permutation(n)              # particle ids scattered over the voxels
    pos = pos[order]
    spec = _spec(n, (1.0, 1.0, 1.0), 0.1, 32)
    b = SceneBatch([spec])
    shuffle = rng.permutation(n)            # and the state in any order
    p4, v4, _, _ = to_device(pos[shuffle], np.zeros((n, 3)))
    pid = torch.as_tensor(shuffle.astype(np.int32), device="cuda")
    vox = K.assign_voxels_to_particles(b, p4).cpu().numpy()
    _, _, ids, _, start, count = K.organize_voxels(b, p4, v4, pid)
    want = shuffle[np.lexsort((shuffle, vox))]
    np.testing.assert_array_equal(ids.cpu().numpy(), want)
    np.testing.assert_array_equal(count.cpu().numpy(), np.bincount(vox, minlength=b.n_voxels))
    b.close()
