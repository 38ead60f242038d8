"""Device memory of the pool of long neighbour lists: 512 bytes per particle of
the scenes that need one, no more, given back when none is left, and counted by
the server's admission."""
import numpy as np
import pytest

from gpu_util import torch_cuda

pytestmark = pytest.mark.gpu

GRAIN = 4 << 20      # two allocation granules


def _free():
    torch = torch_cuda()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


def _used_by(specs):
    """Bytes of a context and its tensors, which are gone when it returns."""
    from sphgb.device import SceneBatch
    before = _free()
    b = SceneBatch(specs)
    used = before - _free()
    b.close()
    return used


def test_pool_is_that_of_the_uncapped_scenes():
    torch_cuda()
    from sphgb.device import SceneBatch
    from sphgb.serve import footprint
    from test_gpu_density_paths import _spec
    n = 400_000
    capped = _spec(n, (5.0, 5.0, 5.0), 0.1, 32)
    small = _spec(2000, (1.0, 1.0, 1.0), 0.1, 0)
    _used_by([capped])      # whatever a first context sets up for good
    base = _used_by([capped])
    # one small uncapped scene costs its own lists, not the capped scene's
    assert _used_by([capped, small]) - base < 2000 * 4096 + GRAIN
    for cap in (0, 33):
        spec = _spec(n, (5.0, 5.0, 5.0), 0.1, cap)
        pool = _used_by([spec]) - base
        assert 512 * n - GRAIN < pool <= footprint(spec) - footprint(capped) + GRAIN
        # reconfigured to capped scenes: the pool is given back
        b = SceneBatch([spec])
        b.reconfigure([capped])
        before = _free()
        b.reconfigure([spec])
        assert 512 * n - GRAIN < before - _free() < 512 * n + GRAIN
        b.close()
        del b


def test_footprint_counts_long_lists():
    from sphgb.serve import footprint
    from test_gpu_density_paths import _spec
    one = {cap: footprint(_spec(1000, (1.0, 1.0, 1.0), 0.1, cap)) for cap in (1, 32, 33, 48, 0)}
    assert one[1] == one[32]
    assert one[33] == one[48] == one[0] == one[32] + 512 * 1000
