"""The step's density passes (tensor-core decisions for sparse and uncapped
scenes, ballots for dense ones) against the thread-per-particle pass, which
walks the reference's way: neighbour rows, counts, densities and the next state
bit for bit, over the forms of scene where the fast passes branch."""
import numpy as np
import pytest

from gpu_util import torch_cuda

pytestmark = pytest.mark.gpu


def _spec(n, space, h, cap, walk="ceil", voxel=None, mass=0.008):
    from sphgb.config import SPHConstants, f32
    from sphgb.data_classes import Pipe, Segment, SimulationParameters
    from sphgb.device import SceneSpec
    params = SimulationParameters(
        particle_count=n, external_force=f32((0.1, -9.81, 0.2)), duration=1, fps=2000.0,
        pipe=Pipe([Segment()]), space_size=f32(space),
        voxel_size=f32(voxel if voxel is not None else (h, h, h)))
    const = SPHConstants(mass=mass, inf_r=float(f32(h)), rho_0=1000.0, k=3.0, visc=3.5, damp=0.5,
                         max_neighbours=cap, walk_dims=walk).rounded()
    return SceneSpec(params, const, 'BOX')


def _both(specs, pos, vel):
    from sphgb import _capi
    from sphgb.device import SceneBatch
    from sphgb.data_classes import SimulationState
    out = []
    for variant in (_capi.DENSITY_WARP, _capi.DENSITY_THREAD):
        b = SceneBatch(specs)
        b.set_tuning(density_variant=variant)
        b.load_states([SimulationState(p, v, np.zeros(len(p))) for p, v in zip(pos, vel)])
        b.step(1)
        lst, cnt = b.step_neighbours()
        out.append([t.cpu().numpy() for t in (b.rho, b.pos, b.vel, b.pid, lst, cnt)])
        b.close()
    for fast, plain, what in zip(*out, ("density", "position", "velocity", "pid", "list", "count")):
        np.testing.assert_array_equal(fast, plain, err_msg=what)
    return out[0]


def _fill(n, space, seed):
    rng = np.random.default_rng(seed)
    pos = rng.random((n, 3), dtype=np.float32) * np.asarray(space, dtype=np.float32)
    vel = rng.standard_normal((n, 3), dtype=np.float32) * np.float32(0.1)
    return pos.astype(np.float64), vel.astype(np.float64)


@pytest.mark.parametrize("cap", [1, 2, 15, 16, 17, 31, 32, 33, 48, 0])
@pytest.mark.parametrize("per_voxel", [0.4, 4.0, 7.5])
def test_caps_and_occupancies(cap, per_voxel):
    torch_cuda()
    h, side = 0.1, 1.0
    n = int(per_voxel * 1000)
    pos, vel = _fill(n, (side,) * 3, seed=cap * 10 + int(per_voxel))
    _both([_spec(n, (side,) * 3, h, cap)], [pos], [vel])


@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 31, 33, 400, 1500])
def test_one_voxel(n):
    """Every particle in one voxel and its corner neighbours: tasks of every
    length, walks of several chunks, and the skip of unreachable voxels."""
    torch_cuda()
    for cap in (32, 0):
        pos, vel = _fill(n, (0.13, 0.12, 0.11), seed=n)
        pos = pos + 0.3
        out = _both([_spec(n, (1.0, 1.0, 1.0), 0.1, cap)], [pos], [vel])
        assert np.isfinite(out[0]).all()


@pytest.mark.parametrize("voxel", [(0.1, 0.1, 0.1), (0.12, 0.1, 0.11), (0.25, 0.25, 0.25),
                                   (0.06, 0.06, 0.06), (0.09, 0.2, 0.1), (0.5, 0.5, 0.5)])
@pytest.mark.parametrize("walk", ["ceil", "truncated"])
@pytest.mark.parametrize("cap", [32, 0])
def test_voxel_sizes(voxel, walk, cap):
    """Voxels that differ from the radius, and walks over the wrong voxels (the
    reference's truncated dims): candidates far from the task's voxel."""
    torch_cuda()
    pos, vel = _fill(3000, (0.95, 0.93, 1.0), seed=3)
    _both([_spec(3000, (0.95, 0.93, 1.0), 0.1, cap, walk, voxel)], [pos], [vel])


@pytest.mark.parametrize("cap", [32, 0])
def test_lattice_at_the_radius(cap):
    """Pairs exactly at the radius or one unit in the last place from it: the
    decisions of the guard band."""
    torch_cuda()
    h = np.float32(0.1)
    g = np.stack(np.meshgrid(*[np.arange(14)] * 3, indexing="ij"), -1).reshape(-1, 3)
    pos = (g * (h / np.float32(2.0)) + np.float32(0.05)).astype(np.float32)
    rng = np.random.default_rng(1)
    nudge = rng.integers(-1, 2, size=pos.shape)
    pos = np.where(nudge < 0, np.nextafter(pos, np.float32(0)),
                   np.where(nudge > 0, np.nextafter(pos, np.float32(9)), pos)).astype(np.float64)
    vel = rng.normal(0, 0.1, pos.shape).astype(np.float32).astype(np.float64)
    _both([_spec(len(pos), (1.0, 1.0, 1.0), float(h), cap)], [pos], [vel])


@pytest.mark.parametrize("cap", [32, 0])
def test_outside_and_non_finite(cap):
    """Particles far outside the box (clamped voxels) and without a finite
    position, among ordinary ones."""
    torch_cuda()
    from sphgb import _capi
    from sphgb.device import SceneBatch
    from sphgb.data_classes import SimulationState
    pos, vel = _fill(2500, (1.0, 1.0, 1.0), seed=9)
    pos[7] = (-3.0, 0.5, 0.5)
    pos[8] = (1.0e6, 0.31, 0.72)
    pos[9] = (0.4, 3.0e30, -2.0e20)
    pos[11, 1] = np.nan
    pos[2400, 2] = np.inf
    specs = [_spec(2500, (1.0, 1.0, 1.0), 0.1, cap)]
    got = []
    for variant in (_capi.DENSITY_WARP, _capi.DENSITY_THREAD):
        b = SceneBatch(specs)
        b.set_tuning(density_variant=variant)
        b.load_states([SimulationState(pos, vel, np.zeros(2500))])
        b.step(1)
        got.append([t.cpu().numpy() for t in b.export_aos_f64()] +
                   [t.cpu().numpy() for t in b.step_neighbours()])
        b.close()
    for a, c in zip(*got):
        np.testing.assert_array_equal(a, c)


def test_mixed_batch():
    """Sparse (tiled), dense (row-major) and truncated scenes in one context:
    both passes run, each on its voxels."""
    torch_cuda()
    rng = np.random.default_rng(5)
    specs, pos, vel = [], [], []
    for n, space, walk in ((3000, (1.0, 1.0, 1.0), "ceil"), (4000, (0.5, 0.5, 0.5), "ceil"),
                           (700, (0.95, 0.95, 0.95), "truncated"), (9000, (0.3, 0.3, 0.4), "ceil")):
        p, v = _fill(n, space, seed=int(rng.integers(1 << 30)))
        specs.append(_spec(n, space, 0.1, 32, walk))
        pos.append(p)
        vel.append(v)
    _both(specs, pos, vel)
