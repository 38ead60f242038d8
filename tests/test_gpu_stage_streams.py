"""Stage calls of one context on several streams share force records and lists:
each call waits for the one before it, whatever stream that was on, so calls
with different inputs that nothing else orders do not disturb each other."""
import numpy as np
import pytest

from gpu_util import to_device, torch_cuda

pytestmark = pytest.mark.gpu


def _inputs(b, n, seeds):
    """Sorted states with their tables, densities and the two calls' results
    from calls that are waited for one by one."""
    torch = torch_cuda()
    from sphgb import kernels as K
    from test_gpu_density_paths import _fill
    steps = torch.zeros(1, dtype=torch.int32, device="cuda")
    cases = []
    for seed in seeds:
        pos, vel = _fill(n, (1.0, 1.0, 1.0), seed=seed)
        p4, v4, pid, _ = to_device(pos, vel)
        pS, vS, idS, _, start, count = K.organize_voxels(b, p4, v4, pid)
        rho = K.density(b, pS, start, count)
        pv = (pS, vS, rho, start, count)
        integ = (pS, vS, rho, idS, start, count, steps)
        torch.cuda.synchronize()
        want = [t.cpu().numpy() for t in K.pressure_viscosity(b, *pv)]
        want += [t.cpu().numpy() for t in K.integrate(b, *integ) if t is not None]
        cases.append((pv, integ, want))
    return cases


def _compare(got, cases):
    torch_cuda().cuda.synchronize()
    for g, (_, _, want) in zip(got, cases):
        for a, c in zip([t for t in g if t is not None], want):
            np.testing.assert_array_equal(a.cpu().numpy(), c)


def test_streams_that_nothing_else_orders():
    torch = torch_cuda()
    from sphgb import kernels as K
    from sphgb.device import SceneBatch
    from test_gpu_density_paths import _spec
    n = 60_000
    b = SceneBatch([_spec(n, (1.0, 1.0, 1.0), 0.05, 32)])
    cases = _inputs(b, n, range(4))
    streams = [torch.cuda.Stream() for _ in cases]
    torch.cuda.synchronize()
    got = [[] for _ in cases]
    for _ in range(3):
        got = [[] for _ in cases]
        for k, (pv, _, _) in enumerate(cases):
            with torch.cuda.stream(streams[k]):
                got[k] += K.pressure_viscosity(b, *pv)
        for k, (_, integ, _) in enumerate(cases):
            with torch.cuda.stream(streams[k]):
                got[k] += K.integrate(b, *integ)
        _compare(got, cases)
    b.close()


def test_streams_that_come_and_go():
    """Every call on a stream of its own, destroyed with the call on it: the next
    stream may have the same handle."""
    torch = torch_cuda()
    import ctypes
    from sphgb import kernels as K
    from sphgb.device import SceneBatch
    from test_gpu_density_paths import _spec
    n = 60_000
    b = SceneBatch([_spec(n, (1.0, 1.0, 1.0), 0.05, 32)])
    cases = _inputs(b, n, range(3))
    rt = torch.cuda.cudart()
    got = [[] for _ in cases]
    for call in (K.pressure_viscosity, K.integrate):
        for k, (pv, integ, _) in enumerate(cases):
            handle = ctypes.c_void_p()
            assert int(rt.cudaStreamCreate(ctypes.addressof(handle))) == 0
            # the outputs belong to the test's own stream, whose memory outlives the call
            got[k] += call(b, *(pv if call is K.pressure_viscosity else integ),
                           stream=torch.cuda.ExternalStream(handle.value))
            assert int(rt.cudaStreamDestroy(handle.value)) == 0
    _compare(got, cases)
    b.close()
