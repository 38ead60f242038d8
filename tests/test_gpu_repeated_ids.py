"""Repeated particle ids (a caller's mistake) stay inside their voxel: the sort
of big voxels orders them like any others, so no particle is written to a slot
of another voxel or past the end of the output."""
import numpy as np
import pytest

from gpu_util import torch_cuda

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [17, 64, 65, 95, 133, 511, 512, 513, 1025])
@pytest.mark.parametrize("twice", ["largest", "middle", "all"])
def test_repeated_ids_stay_in_their_voxel(size, twice):
    torch = torch_cuda()
    from sphgb import _capi
    from sphgb.device import SceneBatch
    from test_gpu_density_paths import _spec
    rng = np.random.default_rng(size)
    sizes = (size, 3, size)          # a voxel behind the first; the last ends the output
    n = sum(sizes)
    vid = np.repeat(np.arange(3), sizes)
    ids = np.concatenate([rng.permutation(m) + 10_000 * v for v, m in enumerate(sizes)])
    for v in (0, 2):
        at = np.flatnonzero(vid == v)
        if twice == "all":
            ids[at] = ids[at[0]]
        else:
            rank = size - 2 if twice == "largest" else size // 2
            low, high = (at[np.argsort(ids[at])[r]] for r in (rank, rank + 1))
            ids[low] = ids[high]
    # the state in any order, the two equal ids of a voxel at any two places
    mix = rng.permutation(n)
    ids, vid = ids[mix], vid[mix]
    pos = np.zeros((n, 4), dtype=np.float32)
    pos[:, :3] = 0.05
    pos[:, 0] += 0.1 * vid
    b = SceneBatch([_spec(n, (0.3, 0.1, 0.1), 0.1, 32)])
    b.set_tuning(big_voxel=16)
    guard = 64
    p4 = torch.as_tensor(pos, device="cuda")
    pid = torch.as_tensor(ids.astype(np.int32), device="cuda")
    pos_o, vel_o = (torch.full((n + guard, 4), -7.0, device="cuda") for _ in range(2))
    pid_o = torch.full((n + guard,), -7, dtype=torch.int32, device="cuda")
    start, count = (torch.empty(b.n_voxels, dtype=torch.int32, device="cuda") for _ in range(2))
    for _ in range(4):                # whatever order the particles arrive in
        for t in (pos_o, vel_o, pid_o):
            t.fill_(-7)
        _capi.call("sphgb_organize_voxels", b.handle, p4.data_ptr(), p4.data_ptr(), pid.data_ptr(),
                   None, pos_o.data_ptr(), vel_o.data_ptr(), pid_o.data_ptr(), None,
                   start.data_ptr(), count.data_ptr(), torch.cuda.current_stream().cuda_stream)
        got = pid_o.cpu().numpy()
        assert (got[n:] == -7).all()
        assert (pos_o[n:].cpu().numpy() == -7).all() and (vel_o[n:].cpu().numpy() == -7).all()
        want = ids[np.lexsort((ids, vid))]
        # equal ids share the first one's slot; every other id is in its place
        first = np.ones(n, dtype=bool)
        first[1:] = want[1:] != want[:-1]
        np.testing.assert_array_equal(got[:n][first], want[first])
        assert (got[:n][~first] == -7).all()
    b.close()
