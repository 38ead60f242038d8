"""The stage entry points build neighbour lists with the step's density passes;
under stream capture they walk, one thread per particle.  Both give the same
bits, also when the table is not that of the state (the lists are then dropped
on the device), and leave the latest step's lists alone."""
import numpy as np
import pytest

from gpu_util import to_device, torch_cuda

pytestmark = pytest.mark.gpu


def _stages(b, pS, vS, idS, start, count, steps):
    from sphgb import kernels as K
    rho = K.density(b, pS, start, count)
    P, V = K.pressure_viscosity(b, pS, vS, rho, start, count)
    return [rho, P, V, *[t for t in K.integrate(b, pS, vS, rho, idS, start, count, steps)
                         if t is not None]]


@pytest.mark.parametrize("n,space,cap,walk", [(1, 1.0, 32, "ceil"), (5000, 1.0, 32, "ceil"),
                                              (6000, 0.4, 32, "ceil"), (5000, 1.0, 0, "ceil"),
                                              (5000, 1.0, 7, "ceil"), (4000, 0.95, 32, "truncated")])
@pytest.mark.parametrize("foreign", [False, True])
def test_lists_equal_walks(n, space, cap, walk, foreign):
    torch = torch_cuda()
    from sphgb import kernels as K
    from sphgb.data_classes import SimulationState
    from sphgb.device import SceneBatch
    from test_gpu_density_paths import _fill, _spec
    pos, vel = _fill(n, (space,) * 3, seed=n + cap)
    b = SceneBatch([_spec(n, (space,) * 3, 0.1, cap, walk)])
    b.load_states([SimulationState(pos, vel, np.zeros(n))])
    b.step(1)
    own = [t.clone() for t in b.step_neighbours()]
    p4, v4, pid, _ = to_device(pos, vel)
    pS, vS, idS, _, start, count = K.organize_voxels(b, p4, v4, pid)
    if foreign:       # the state moves on, the table stays
        pS = pS.clone()
        pS[:, :3] = (pS[:, :3] + 0.07) % space
    steps = torch.zeros(1, dtype=torch.int32, device="cuda")
    with_lists = [t.clone() for t in _stages(b, pS, vS, idS, start, count, steps)]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        walked = _stages(b, pS, vS, idS, start, count, steps)
    graph.replay()
    torch.cuda.synchronize()
    for a, c in zip(with_lists, walked):
        np.testing.assert_array_equal(a.cpu().numpy(), c.cpu().numpy())
    for a, c in zip(own, b.step_neighbours()):
        np.testing.assert_array_equal(a.cpu().numpy(), c.cpu().numpy())
    # another stream: ordered behind the first by the context
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        again = _stages(b, pS, vS, idS, start, count, steps)
    side.synchronize()
    for a, c in zip(with_lists, again):
        np.testing.assert_array_equal(a.cpu().numpy(), c.cpu().numpy())
    b.close()
