"""The host call's direct slot order (kernels read and write the host buffers)
against the device path: ordinary and page-locked buffers, at offsets that are
8-byte aligned only, in place, and on both sides of its size limits."""
import numpy as np
import pytest

from gpu_util import torch_cuda

pytestmark = pytest.mark.gpu


def _buffer(shape, pinned, offset):
    torch = torch_cuda()
    n = int(np.prod(shape)) + offset
    flat = (torch.empty(n, dtype=torch.float64, pin_memory=True).numpy() if pinned
            else np.empty(n))
    return flat[offset:].reshape(shape)


@pytest.mark.parametrize("n", [1, 255, 257, 5000, 40_000, 40_001, 131_073])
@pytest.mark.parametrize("pinned", [False, True])
@pytest.mark.parametrize("in_place", [False, True])
def test_slot_order_equals_device_path(n, pinned, in_place):
    torch_cuda()
    from sphgb import _capi
    from sphgb.data_classes import SimulationState
    from sphgb.device import SceneBatch
    from test_gpu_density_paths import _fill, _spec
    pos, vel = _fill(n, (1.0, 1.0, 1.0), seed=n)
    spec = _spec(n, (1.0, 1.0, 1.0), 0.05, 32, mass=0.001)
    b = SceneBatch([spec])
    b.load_states([SimulationState(pos, vel, np.zeros(n))])
    b.step(1)
    want = [t.cpu().numpy() for t in b.export_aos_f64()]
    b.close()
    b = SceneBatch([spec])
    b.set_host_order(_capi.HOST_ORDER_SLOT)
    bufs = [_buffer(s, pinned, 1) for s in ((n, 3), (n, 3), (n, 3), (n, 3), (n,))]
    if in_place:
        bufs[2], bufs[3] = bufs[0], bufs[1]
    bufs[0][...], bufs[1][...] = pos, vel
    got = b.compute_next_state_host(*bufs)
    for g, w in zip(got, want):
        np.testing.assert_array_equal(g, w)
    b.close()
