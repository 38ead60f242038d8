"""Host buffers at addresses that are no multiple of 8 (arrays that view packed
bytes): the host call copies them, whatever their size, instead of letting
kernels read and write them."""
import numpy as np
import pytest

from gpu_util import torch_cuda

pytestmark = pytest.mark.gpu


def _buffer(shape, pinned, offset):
    torch = torch_cuda()
    n = 8 * int(np.prod(shape))
    raw = (torch.empty(n + offset, dtype=torch.uint8, pin_memory=True).numpy() if pinned
           else np.empty(n + offset, dtype=np.uint8))
    return raw[offset:].view(np.float64).reshape(shape)


@pytest.mark.parametrize("n", [1, 3000])
@pytest.mark.parametrize("pinned", [False, True])
@pytest.mark.parametrize("which", [0, 1, 2, 3, 4])
def test_any_byte_address(n, pinned, which):
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
    for order in (_capi.HOST_ORDER_AUTO, _capi.HOST_ORDER_SLOT):
        b = SceneBatch([spec])
        b.set_host_order(order)
        bufs = [_buffer(s, pinned, 4 if k == which else 8)
                for k, s in enumerate(((n, 3), (n, 3), (n, 3), (n, 3), (n,)))]
        assert bufs[which].ctypes.data % 8 == 4
        bufs[0][...], bufs[1][...] = pos, vel
        for g, w in zip(b.compute_next_state_host(*bufs), want):
            np.testing.assert_array_equal(g, w)
        b.close()
