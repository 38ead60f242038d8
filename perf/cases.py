"""The calls of a user of this package that its speed is judged by, with their inputs.

Four ways of using the package, over the range of sizes that its scenes, tests
and benchmark cover (1,024 to 4,194,304 particles):

* ``device``: a state that lives on the GPU.  FP64 rows in particle order go in
  (SceneBatch.load_aos_device), one step or a run of steps in a CUDA graph
  follows, the result is the bound state (slot order, particle ids beside it).
  A run of steps is what a simulation does between two frames.
* ``batch``: many independent boxes in one context, advanced by one graph.
* ``host``: the reference's own boundary, compute_next_state on FP64 host
  arrays: GB300SPHStrategy on ordinary numpy arrays (``pinned`` false), or the
  same call on page-locked buffers that the caller keeps (``pinned`` true).
* ``stages``: the reference's kernels one by one (sphgb.kernels).

Scenes: ``box`` is the jittered dam-break block (2.25 spacings of smoothing
radius, about 11 particles per voxel, so the cap of 32 neighbours binds), with
ids in lattice order or shuffled (``shuffle``), as they are once a fluid has
mixed; ``pipe`` is the pipe flow's start state (about 133 particles per voxel,
FP64 wall response), scaled to other sizes with its neighbour count kept.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "cuda-sph_gb300"))

from sphgb import kernels, scenes                          # noqa: E402
from sphgb.config import f32                               # noqa: E402
from sphgb.data_classes import SimulationState             # noqa: E402
from sphgb.device import SceneBatch                        # noqa: E402
from sphgb.strategies import GB300SPHStrategy              # noqa: E402

DEV = "cuda"


def _box(name, use, nx, ny, nz, steps=1, cap=32, walk="ceil", shuffle=False, pinned=False,
         fine=False):
    """One box.  ``fine``: the 4,194,304-particle benchmark's spacing, radius
    and 2 m box instead of the 0.02 m spacing of the small dam break."""
    c = dict(use=use, scene="box", nx=nx, ny=ny, nz=nz, steps=steps, cap=cap, walk=walk,
             shuffle=shuffle, pinned=pinned, fine=fine)
    return c if name is None else dict(c, name=name)


def _pipe(name, use, n, steps=1, pinned=False):
    c = dict(use=use, scene="pipe", n=n, steps=steps, pinned=pinned)
    return c if name is None else dict(c, name=name)


def _batch(name, scenes_n, n_min, n_max, steps):
    c = dict(use="batch", scene="boxes", scenes=scenes_n, n_min=n_min, n_max=n_max, steps=steps)
    return c if name is None else dict(c, name=name)


def listed():
    return [
        # the smallest scene anybody steps, one call at a time
        _box("box_1k", "device", 8, 16, 8),
        # the small dam break between two frames: 50 short steps in a graph
        _box("box_8k_run", "device", 16, 32, 16, steps=50),
        # odd sizes, ids scattered over space as in a mixed fluid
        _box("box_odd_52k", "device", 37, 61, 23, shuffle=True),
        # an ordinary simulation, several steps per frame
        _box("box_262k_run", "device", 64, 64, 64, steps=8),
        # the benchmark's scene, the largest
        _box("box_4m", "device", 128, 256, 128, fine=True),
        # no neighbour cap: the physics without the reference's cut at 32
        _box("box_uncapped_33k", "device", 32, 32, 32, cap=0),
        # dense voxels and the FP64 wall response
        _pipe("pipe_262k", "device", 262_144),
        # independent scenes of mixed sizes side by side (parameter studies, serving)
        _batch("batch_48", 48, 1024, 65_536, steps=10),
        # the drop-in call with ordinary numpy arrays: small, and the pipe
        _box("host_box_8k", "host", 16, 32, 16),
        _pipe("host_pipe_262k", "host", 262_144),
        # the drop-in call at full size on page-locked buffers
        _box("host_box_4m", "host", 128, 256, 128, pinned=True, fine=True),
        # the reference's kernels called one by one
        _box("stages_111k", "stages", 48, 48, 48),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _block(rng, lo, hi):
    """Lattice sides of a block of about log-uniform size, not cubic."""
    n = _log(rng, lo, hi)
    a = n ** (1.0 / 3.0)
    nx = max(4, int(round(a * rng.uniform(0.6, 1.3))))
    nz = max(4, int(round(a * rng.uniform(0.6, 1.3))))
    return nx, max(4, int(round(n / (nx * nz)))), nz


def draw(rng):
    use = rng.choice(["device", "device", "device", "pipe", "batch", "host", "host", "stages"])
    if use == "device":
        nx, ny, nz = _block(rng, 1024, 2_000_000)
        few = nx * ny * nz > 300_000
        # the fine scene and the cut walk blow up within a few steps: one step
        fine = few and rng.random() < 0.5
        walk = rng.choice(["ceil", "ceil", "ceil", "truncated"])
        once = fine or walk == "truncated"
        return _box(None, "device", nx, ny, nz,
                    steps=1 if once else rng.choice([1, 3] if few else [1, 4, 16]),
                    cap=rng.choice([32, 32, 32, 24, 0]), walk=walk,
                    shuffle=rng.random() < 0.4, fine=fine)
    if use == "pipe":
        return _pipe(None, "device", int(_log(rng, 2048, 300_000)))
    if use == "batch":
        lo = int(_log(rng, 1024, 8192))
        return _batch(None, rng.randint(3, 48), lo, int(lo * _log(rng, 1.5, 8)), rng.randint(2, 10))
    if use == "host":
        if rng.random() < 0.35:
            return _pipe(None, "host", int(_log(rng, 2048, 300_000)), pinned=rng.random() < 0.5)
        nx, ny, nz = _block(rng, 1024, 1_000_000)
        return _box(None, "host", nx, ny, nz, shuffle=rng.random() < 0.4,
                    pinned=rng.random() < 0.5)
    nx, ny, nz = _block(rng, 1024, 262_144)
    return _box(None, "stages", nx, ny, nz, cap=rng.choice([32, 32, 16, 0]),
                shuffle=rng.random() < 0.4)


# ---- inputs -----------------------------------------------------------------

def _scene(case, seed):
    """(spec, FP32-representable FP64 positions, velocities) of a one-scene case."""
    rng = np.random.default_rng([int(seed), 77])
    if case["scene"] == "pipe":
        n = case["n"]
        h = 0.02 if n == 262_144 else 0.02 * (262_144 / n) ** (1.0 / 3.0)
        spec, st = scenes.pipe_flow(n=n, h=h, seed=int(seed))
        return spec, st.position, st.velocity
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    if case["fine"]:
        edge = max(2.0, 1.25 * 0.005 * max(nx, ny, nz))
        kw = dict(spacing=0.005, jitter=0.0005, h=0.0112, mass=1.25e-4)
    else:
        edge = max(1.0, 1.25 * 0.02 * max(nx, ny, nz))
        kw = {}
    spec, st = scenes.box_dam_break(nx=nx, ny=ny, nz=nz, box=(edge, edge, edge), seed=int(seed),
                                    max_neighbours=case["cap"], walk_dims=case["walk"], **kw)
    pos = st.position
    if case["shuffle"]:
        pos = np.ascontiguousarray(pos[rng.permutation(len(pos))])
    # a fluid in motion: a common stream and a spread about it
    vel = rng.standard_normal(pos.shape, dtype=np.float32) * np.float32(0.05)
    vel[:, 0] += np.float32(0.2)
    return spec, pos, vel.astype(np.float64)


def _boxes(case, seed):
    """Boxes of log-uniform sizes, edges 0.5 to 2, gravity in any direction."""
    rng = np.random.default_rng([int(seed), 78])
    # the sizes belong to the case, the particles to the seed
    sizes = np.random.default_rng([case["scenes"], case["n_min"], case["n_max"]])
    specs, pos, vel = [], [], []
    for _ in range(case["scenes"]):
        n = math.exp(sizes.uniform(math.log(case["n_min"]), math.log(case["n_max"])))
        edge, g = sizes.uniform(0.5, 2.0), sizes.normal(size=3)
        nx = max(2, int(round((n / 2.0) ** (1.0 / 3.0))))
        s = min(0.02, 0.9 * edge / (2 * nx))
        spec, st = scenes.box_dam_break(nx=nx, ny=2 * nx, nz=nx, spacing=s, jitter=s / 10.0,
                                        box=(edge, edge, edge), h=1.93 * s, mass=1000.0 * s ** 3,
                                        gravity=tuple(9.81 * g / np.linalg.norm(g)),
                                        seed=int(rng.integers(1 << 31)))
        specs.append(spec)
        pos.append(st.position)
        vel.append(f32(rng.normal(0.0, 0.05, size=st.position.shape)))
    return specs, np.concatenate(pos), np.concatenate(vel)


def _pinned(a):
    t = torch.empty(a.shape, dtype=torch.float64, pin_memory=True)
    t.numpy()[...] = a
    return t.numpy(), t


def prepare(case, seed):
    use = case["use"]
    st = {"use": use, "steps": case.get("steps", 1)}
    if use == "batch":
        specs, pos, vel = _boxes(case, seed)
    else:
        spec, pos, vel = _scene(case, seed)
        specs = [spec]
    n = len(pos)
    if use in ("device", "batch"):
        st["scenes"] = SceneBatch(specs, device=DEV)
        st["pos"] = torch.from_numpy(np.ascontiguousarray(pos)).to(DEV)
        st["vel"] = torch.from_numpy(np.ascontiguousarray(vel)).to(DEV)
    elif use == "host":
        if case["pinned"]:
            st["scenes"] = SceneBatch(specs, device=DEV)
            bufs = [_pinned(a) for a in (pos, vel, np.zeros((n, 3)), np.zeros((n, 3)), np.zeros(n))]
            st["bufs"], st["keep"] = [b[0] for b in bufs], [b[1] for b in bufs]
        else:
            st["strategy"] = GB300SPHStrategy(specs[0].params, specs[0].constants, specs[0].mode,
                                              device=DEV)
            st["state"] = SimulationState(pos, vel, np.zeros(n))
    else:
        st["scenes"] = SceneBatch(specs, device=DEV)
        four = np.zeros((n, 4), dtype=np.float32)
        four[:, :3] = pos
        st["pos"] = torch.from_numpy(four.copy()).to(DEV)
        four[:, :3] = vel
        st["vel"] = torch.from_numpy(four).to(DEV)
        st["pid"] = torch.arange(n, dtype=torch.int32, device=DEV)
        st["step_no"] = torch.zeros(1, dtype=torch.int32, device=DEV)
    return st


def run(state):
    use = state["use"]
    if use in ("device", "batch"):
        b = state["scenes"]
        b.load_aos_device(state["pos"], state["vel"])
        b.step(state["steps"], use_graph=state["steps"] > 1)
        return [b.pos, b.vel, b.rho, b.pid] + ([b.pos64] if b.any_pipe else [])
    if use == "host":
        if "strategy" in state:
            new = state["strategy"].compute_next_state(state["state"])
            return [new.position, new.velocity, new.density]
        return list(state["scenes"].compute_next_state_host(*state["bufs"]))
    b = state["scenes"]
    pos, vel, pid, _, start, count = kernels.organize_voxels(b, state["pos"], state["vel"],
                                                             state["pid"])
    rho = kernels.density(b, pos, start, count)
    p, v = kernels.pressure_viscosity(b, pos, vel, rho, start, count)
    pos_n, vel_n, pid_n, _, force = kernels.integrate(b, pos, vel, rho, pid, start, count,
                                                      state["step_no"])
    return [pid, start, count, rho, p, v, pos_n, vel_n, pid_n, force]


def _count(case):
    if case["scene"] == "pipe":
        return case["n"]
    if case["scene"] == "box":
        return case["nx"] * case["ny"] * case["nz"]
    sizes = np.random.default_rng([case["scenes"], case["n_min"], case["n_max"]])
    n = 0
    for _ in range(case["scenes"]):
        t = math.exp(sizes.uniform(math.log(case["n_min"]), math.log(case["n_max"])))
        sizes.uniform(0.5, 2.0), sizes.normal(size=3)
        n += 2 * max(2, int(round((t / 2.0) ** (1.0 / 3.0)))) ** 3
    return n


def work(case):
    """Bytes: FP64 rows in (48 B), and out the float4 state, density and id (40 B;
    FP64 rows, 56 B, from the host call; per further step the state in and out,
    72 B).  Flops: 31 neighbours with a squared distance (8), a density term (5)
    and the pressure and viscosity sums (32) each."""
    n, steps = _count(case), case.get("steps", 1)
    out = {"host": 56, "stages": 40 + 52}.get(case["use"], 40)
    inn = 36 if case["use"] == "stages" else 48
    return {"bytes": float(n) * (inn + out + 72 * (steps - 1)), "flops": float(n) * steps * 31 * 45}


# ---- the same results in 64 bits ---------------------------------------------

def _step64(spec, pos, vel):
    """One step of a scene in FP64, plain torch: (density, pressure, viscosity,
    force, next position, next velocity) in particle order, the voxel
    coordinates and the table's dims.  The walk visits the 27 voxels with x
    outermost and z innermost, a voxel's particles by id, and takes the first
    max_neighbours within the smoothing radius, the particle itself among them."""
    par, c = spec.params, spec.constants.rounded()
    t64 = lambda a: torch.as_tensor(np.asarray(f32(a)), dtype=torch.float64, device=DEV)  # noqa: E731
    space, vs, ext = t64(par.space_size), t64(par.voxel_size), t64(par.external_force)
    q = (np.asarray(f32(par.space_size)) / np.asarray(f32(par.voxel_size)))
    dims = [max(1, int(math.ceil(x))) for x in q]
    wdims = [int(x) for x in q] if c.walk_dims == "truncated" else dims
    dt, h = float(f32(1.0 / float(par.fps))), c.inf_r
    x = torch.as_tensor(pos, dtype=torch.float64, device=DEV)
    v = torch.as_tensor(vel, dtype=torch.float64, device=DEV)
    n = x.shape[0]
    vox = torch.minimum((x / vs).floor().to(torch.int64),
                        torch.tensor(dims, device=DEV) - 1).clamp_(min=0)
    vid = vox[:, 0] + vox[:, 1] * dims[0] + vox[:, 2] * dims[0] * dims[1]
    order = torch.argsort(vid, stable=True)
    nv = max(dims[0] * dims[1] * dims[2], 1)
    count = torch.bincount(vid, minlength=nv)
    start = torch.cumsum(count, 0) - count
    cap = c.max_neighbours if c.max_neighbours > 0 else 1 << 30
    w = 315.0 / (64.0 * math.pi * h ** 9)
    gw, lw = -45.0 / (math.pi * h ** 6), 45.0 / (math.pi * h ** 6)
    x0, x1, x2 = (x[:, a].contiguous() for a in range(3))
    v0, v1, v2 = (v[:, a].contiguous() for a in range(3))
    me = torch.arange(n, device=DEV)

    def walk(visit):
        """visit(i, j, dx, dy, dz, r2) per round of accepted pairs (no i twice)."""
        seen = torch.zeros(n, dtype=torch.int64, device=DEV)
        for a in (-1, 0, 1):
            for b in (-1, 0, 1):
                for d in (-1, 0, 1):
                    k0, k1, k2 = vox[:, 0] + a, vox[:, 1] + b, vox[:, 2] + d
                    ok = ((k0 >= 0) & (k0 < wdims[0]) & (k1 >= 0) & (k1 < wdims[1]) &
                          (k2 >= 0) & (k2 < wdims[2]))
                    nb = torch.where(ok, k0 + k1 * wdims[0] + k2 * wdims[0] * wdims[1],
                                     torch.zeros_like(k0))
                    cnt = torch.where(ok, count[nb], torch.zeros_like(nb))
                    first = start[nb]
                    live = me[cnt > 0]
                    m = 0
                    while live.numel():
                        j = order[first[live] + m]
                        dx, dy, dz = x0[live] - x0[j], x1[live] - x1[j], x2[live] - x2[j]
                        r2 = dx * dx + dy * dy + dz * dz
                        near = (r2.sqrt() <= h) & (seen[live] < cap)
                        i = live[near]
                        seen[i] += 1
                        other = j[near] != i
                        visit(i[other], j[near][other], dx[near][other], dy[near][other],
                              dz[near][other], r2[near][other])
                        m += 1
                        live = live[(cnt[live] > m) & (seen[live] < cap)]

    rho = torch.zeros(n, dtype=torch.float64, device=DEV)

    def add_density(i, j, dx, dy, dz, r2):
        rho[i] += c.mass * (w * (h * h - r2) ** 3)

    walk(add_density)
    press = torch.zeros(3, n, dtype=torch.float64, device=DEV)
    visc = torch.zeros(3, n, dtype=torch.float64, device=DEV)
    fac = c.k * (rho - c.rho_0) / (rho * rho)

    def add_forces(i, j, dx, dy, dz, r2):
        r = r2.sqrt()
        g = (fac[i] + fac[j]) * gw * (h - r) ** 2 / r
        s = c.mass * c.visc / rho[j] * (lw * (h - r)) / rho[i]
        for a, (d, u) in enumerate(((dx, v0), (dy, v1), (dz, v2))):
            press[a][i] += g * d
            visc[a][i] += s * (u[j] - u[i])

    walk(add_forces)
    press, visc = press.t(), visc.t().clamp(max=1.0)
    force = ext - press + visc
    vn = v + force / rho[:, None] * dt
    xn = x + vn * dt
    low, high = xn < 0, xn > space
    xb = torch.where(low, torch.full_like(xn, 1e-3), torch.where(high, space - 1e-3, xn))
    vb = torch.where(low | high, -vn * c.damp, vn)
    return rho, press, visc, force, xb, vb, vox, dims


def _slot_order(spec, vox, dims, stages):
    """Particle at each slot: by voxel, then id.  The step numbers the voxels of
    sparse scenes (at most 8 particles per voxel) in 4x4x4 tiles, x fastest."""
    n = vox.shape[0]
    q = np.asarray(f32(spec.params.space_size)) / np.asarray(f32(spec.params.voxel_size))
    cut = spec.constants.walk_dims == "truncated" and any(int(a) != d for a, d in zip(q, dims))
    x, y, z = vox[:, 0], vox[:, 1], vox[:, 2]
    if stages or cut or n > 8 * dims[0] * dims[1] * dims[2]:
        key = x + y * dims[0] + z * dims[0] * dims[1]
    else:
        t0, t1 = (dims[0] + 3) // 4, (dims[1] + 3) // 4
        tile = ((z // 4) * t1 + y // 4) * t0 + x // 4
        key = tile * 64 + (z % 4) * 16 + (y % 4) * 4 + x % 4
    return torch.argsort(key, stable=True)


def _four(a):
    return torch.cat([a, torch.zeros_like(a[:, :1])], dim=1)


def exact(case, seed):
    """None for runs of several steps: the capped walk makes them chaotic (one
    pair crossing the radius changes who is the 32nd neighbour), so 64 bits say
    nothing about them.  The pipe's wall response is left out (its respawn draws
    random numbers): its densities only."""
    if case.get("steps", 1) > 1 or case["use"] == "batch":
        return None
    spec, pos, vel = _scene(case, seed)
    rho, press, visc, force, xn, vn, vox, dims = _step64(spec, pos, vel)
    pipe = case["scene"] == "pipe"
    if case["use"] == "host":
        return [None, None, rho] if pipe else [xn, vn, rho]
    o = _slot_order(spec, vox, dims, case["use"] == "stages")
    if case["use"] == "stages":
        return [None, None, None, rho[o], _four(press[o]), _four(visc[o]), _four(xn[o]),
                _four(vn[o]), None, _four(force[o])]
    if pipe:
        return [None, None, rho[o], None, None]
    return [_four(xn[o]), _four(vn[o]), rho[o], None]
