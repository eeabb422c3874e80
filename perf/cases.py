"""What the performance of this framework is measured on: time steps of single scenes and of a batch of scenes,
the stand-alone radix sort and the headless renderer, each through its public entry points.

A pass of a scene is what a program does that couples the solver to its own code: hand over positions and velocities,
advance the scene, take the state back. Every pass starts from the same state, so passes can be repeated. The states are
built from the seed: lattices near the rest spacing with a random displacement of each particle, in the velocity field of
the stage of the flow that the case stands for (a column at rest, a collapsing column, a falling sphere at impact), in the
order in which the solver hands a state back (sorted by grid bucket).
"""
import math

import numpy as np
import torch

from pcisph_gb300 import Fluid, setup_scene
from pcisph_gb300 import render as rendering
from pcisph_gb300.batch import Batch
from pcisph_gb300.fluid import RadixSort
from pcisph_gb300.scenes import Scene

DEV = "cuda:0"


def listed():
    return [
        # the smallest scene in use (an interactive demo, a unit of a parameter study): launches and latency
        {"name": "dam_4k", "kind": "dam", "nx": 16, "ny": 16, "nz": 16, "spacing": 0.02, "gap": 1.0, "delta_t": 1e-3,
         "jitter": 0.05, "speed": 0.0, "steps": 1, "iterations": 7, "memory": "device"},
        # the 32,768-particle dam break, a few steps of the collapsing column per exchange with the host program
        {"name": "dam_32k", "kind": "dam", "nx": 32, "ny": 32, "nz": 32, "spacing": 0.02, "gap": 1.01, "delta_t": 1e-3,
         "jitter": 0.15, "speed": 0.5, "steps": 4, "iterations": 6, "memory": "device"},
        # a mid-size column of odd dimensions whose state lives in pinned host memory (a host-side coupling)
        {"name": "dam_157k_host", "kind": "dam", "nx": 67, "ny": 53, "nz": 44, "spacing": 0.01, "gap": 1.01, "delta_t": 5e-4,
         "jitter": 0.15, "speed": 0.8, "steps": 1, "iterations": 6, "memory": "host"},
        # the flagship size: 128 x 128 x 64 particles, the column collapsing
        {"name": "dam_1m", "kind": "dam", "nx": 128, "ny": 128, "nz": 64, "spacing": 0.005, "gap": 1.01, "delta_t": 2.5e-4,
         "jitter": 0.15, "speed": 1.0, "steps": 1, "iterations": 6, "memory": "device"},
        # a sphere of fluid as it hits its pool at 3.1 m/s: its predictions outrun the neighbour lists
        {"name": "drop_100k", "kind": "drop", "count": 99768, "spacing": 0.01, "gap": 1.0, "delta_t": 1e-3, "jitter": 0.05,
         "height": 0.0, "steps": 1, "iterations": 50, "memory": "device"},
        # fluid in a tank of boundary particles, the size of the reference's voxel dam break, 3 to 7 iterations
        {"name": "tank_280k", "kind": "tank", "nx": 96, "ny": 54, "nz": 54, "spacing": 0.01, "gap": 1.0, "delta_t": 5e-4,
         "jitter": 0.05, "speed": 0.5, "steps": 1, "iterations": 7, "memory": "device"},
        # the same at the flagship size: 1,048,576 fluid and about 284,000 boundary particles
        {"name": "tank_1m", "kind": "tank", "nx": 128, "ny": 128, "nz": 64, "spacing": 0.005, "gap": 1.0, "delta_t": 2.5e-4,
         "jitter": 0.05, "speed": 0.5, "steps": 1, "iterations": 7, "memory": "device"},
        # the largest scene: two blocks of 4,194,304 particles, the first step, which takes every iteration it may
        {"name": "blocks_8m", "kind": "blocks", "nx": 256, "ny": 128, "nz": 128, "spacing": 0.0025, "gap": 1.0,
         "delta_t": 1.25e-4, "jitter": 0.05, "speed": 0.0, "steps": 1, "iterations": 50, "memory": "device"},
        # a batch of independent scenes (a parameter study, a rollout server), read back every 16 steps
        {"name": "batch_32", "kind": "batch", "scenes": 32, "least": 4096, "most": 131072, "spacing": 0.01, "gap": 1.0,
         "delta_t": 1e-3, "jitter": 0.05, "steps": 16, "iterations": 5},
        # the stable radix sort on its own: 32-bit keys with payloads
        {"name": "sort_3m", "kind": "sort", "count": 3000001, "bits": 32},
        # a frame of the 1M scene
        {"name": "frame_1m", "kind": "frame", "nx": 128, "ny": 128, "nz": 64, "spacing": 0.005, "gap": 1.0, "jitter": 0.1,
         "width": 1280, "height": 720},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _sides(rng, n):
    a, c = rng.uniform(0.6, 2.0), rng.uniform(0.6, 1.6)
    ny = max(6, round((n / (a * c)) ** (1 / 3)))
    return max(6, round(a * ny)), ny, max(6, round(c * ny))


def draw(rng):
    kind = rng.choice(["dam", "dam", "dam", "drop", "tank", "tank", "batch", "sort", "frame"])
    if kind == "sort":
        return {"kind": kind, "count": int(_log(rng, 2e3, 2e7)) | 1, "bits": rng.choice([13, 17, 20, 24, 32])}
    if kind == "batch":
        return {"kind": kind, "scenes": rng.randint(3, 32), "least": 4096, "most": int(_log(rng, 20000, 131072)),
                "spacing": 0.01, "gap": 1.0, "delta_t": 1e-3, "jitter": 0.05, "steps": rng.randint(4, 16), "iterations": 5}
    d = 0.02 * rng.choice([1.0, 0.5, 0.25])
    case = {"kind": kind, "spacing": d, "gap": 1.0, "jitter": rng.uniform(0.04, 0.07)}
    if kind == "frame":
        nx, ny, nz = _sides(rng, _log(rng, 4e3, 1e6))
        return {**case, "nx": nx, "ny": ny, "nz": nz, "width": rng.choice([320, 641, 1280, 1920]), "height": rng.choice([240, 480, 721])}
    if kind == "drop":
        return {**case, "count": int(_log(rng, 8e3, 2.5e5)), "spacing": 0.01, "delta_t": 1e-3, "height": rng.uniform(0.0, 0.4),
                "steps": 1, "iterations": 30, "memory": "device"}
    nx, ny, nz = _sides(rng, _log(rng, 3e3, 1.2e6 if kind == "dam" else 6e5))
    if kind == "dam":
        case.update(gap=1.01, jitter=rng.uniform(0.05, 0.18))
    return {**case, "nx": nx, "ny": ny, "nz": nz, "delta_t": 0.05 * d, "speed": rng.uniform(0.0, 1.0), "steps": 1,
            "iterations": 6 if kind == "dam" else 7, "memory": rng.choice(["device", "device", "host"])}


# ---------------------------------------------------------------------------------------------- inputs


def _generator(seed, part=0):
    g = torch.Generator(device=DEV)
    g.manual_seed((int(seed) * 1000003 + part) % (1 << 62))
    return g


def _block(nx, ny, nz, d, origin, jitter, g):
    """nx * ny * nz particles at cell centres of a lattice of spacing d, x fastest, displaced by up to jitter * d."""
    z, y, x = torch.meshgrid(*(torch.arange(k, device=DEV, dtype=torch.float64) for k in (nz, ny, nx)), indexing="ij")
    p = torch.stack([x.reshape(-1), y.reshape(-1), z.reshape(-1)], 1) + 0.5
    p += (2.0 * torch.rand(p.shape, generator=g, device=DEV, dtype=torch.float64) - 1.0) * jitter
    return p * d + torch.tensor(origin, device=DEV, dtype=torch.float64)


def _collapse(pos, speed, g):
    """The velocities of a column that collapses along x: spreading at its foot, sinking at its top, slightly uneven."""
    size = pos.max(0).values.clamp_min(1e-6)
    q = pos / size
    v = torch.zeros_like(pos)
    v[:, 0] = speed * q[:, 0] * (1.0 - 0.5 * q[:, 1])
    v[:, 1] = -speed * q[:, 1] * (0.3 + 0.7 * q[:, 0])
    return v + 0.02 * speed * (2.0 * torch.rand(v.shape, generator=g, device=DEV, dtype=torch.float64) - 1.0)


def _tank_walls(box, d, layers=2):
    """Boundary particles: sheets of spacing d below the floor and outside the four walls of [0, box]."""
    n = [int(round(b / d)) for b in box]
    z, y, x = torch.meshgrid(torch.arange(n[2] + 2 * layers, device=DEV), torch.arange(n[1] + layers, device=DEV),
                             torch.arange(n[0] + 2 * layers, device=DEV), indexing="ij")
    x, y, z = x.reshape(-1) - layers, y.reshape(-1) - layers, z.reshape(-1) - layers
    wall = (x < 0) | (x >= n[0]) | (y < 0) | (z < 0) | (z >= n[2])
    p = torch.stack([x[wall], y[wall], z[wall]], 1).to(torch.float64)
    return ((p + 0.5) * d).float().contiguous()


def _drop(count, d, height, jitter, g):
    """A sphere of 70% of the particles, `height` above a pool of the rest, after falling from 0.5 m above it."""
    n_sphere = int(round(0.7 * count))
    n_pool = count - n_sphere
    radius = (3.0 * n_sphere / (4.0 * math.pi)) ** (1.0 / 3.0) * d
    depth = max(2 * d, 0.5 * radius)
    side = max(4, int(round(math.sqrt(n_pool * d / depth))), int(math.ceil(2.0 * radius / d)) + 2)
    layers = max(1, int(round(n_pool / (side * side))))
    pool = _block(side, layers, side, d, (0.0, 0.0, 0.0), jitter, g)
    top = layers * d + height + 0.5 * d
    centre = torch.tensor([0.5 * side * d, top + radius, 0.5 * side * d], device=DEV, dtype=torch.float64)
    m = int(math.ceil(radius / d)) + 1
    cube = _block(2 * m, 2 * m, 2 * m, d, (float(centre[0]) - m * d, float(centre[1]) - m * d, float(centre[2]) - m * d), 0.0, g)
    sphere = cube[(cube - centre).norm(dim=1) <= radius]
    sphere = sphere + (2.0 * torch.rand(sphere.shape, generator=g, device=DEV, dtype=torch.float64) - 1.0) * jitter * d
    pos = torch.cat([pool, sphere])
    vel = torch.zeros_like(pos)
    vel[pool.shape[0]:, 1] = -math.sqrt(2.0 * 9.81 * max(0.0, 0.5 - height))
    return pos, vel, (side * d, layers * d + 0.5 + 2.0 * radius + 2 * d, side * d)


def _f32(v):
    return float(np.float32(v))


def _cells(x, h):
    """Grid cells of float32 positions: floor of the float32 quotient."""
    return torch.floor(x / torch.full((1, 3), h, dtype=torch.float32, device=x.device)).to(torch.int64)


def _bucket(c, buckets):
    m = 0xFFFFFFFF
    h = ((c[:, 0] * 19349663) & m) ^ ((c[:, 1] * 73856093) & m) ^ ((c[:, 2] * 83492791) & m)
    v = ((h << 6) & m) + (c[:, 0] & 63) + 4 * (c[:, 1] & 63) + 16 * (c[:, 2] & 63)
    return (v & 0x7FFFFFFF) % buckets


def _kernel_radius(d):
    return float(np.float32(4) * np.float32(0.5 * d))


def _buckets(n):
    return max(64, n // 2 - n // 2 % 64)


def _scene(case, seed):
    """(scene, positions, velocities) of a single-scene case: float32 (n, 3) on the GPU."""
    g, d = _generator(seed), case["spacing"]
    walls, limits = torch.zeros((0, 3), device=DEV), (3, 50)
    if case["kind"] == "drop":
        pos, vel, box = _drop(case["count"], d, case["height"], case["jitter"], g)
    else:
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        # `gap`: a little apart, as the column is once its first steps have relaxed it; 1: the scene as it is set up
        pos = _block(nx, ny, nz, d, (0.0, 0.0, 0.0), case["jitter"], g) * case["gap"]
        vel = _collapse(pos, case.get("speed", 0.0), g)
        box = (2.5 * nx * d, 2.0 * ny * d, nz * d)
        if case["kind"] == "blocks":
            far = _block(nx, ny, nz, d, (1.5 * nx * d, 0.0, 0.0), case["jitter"], g) * case["gap"]
            pos, vel = torch.cat([pos, far]), torch.cat([vel, torch.zeros_like(far)])
        if case["kind"] == "tank":
            box = (2.0 * nx * d, 1.5 * ny * d, nz * d)
            walls, limits = _tank_walls(box, d), (3, 7)
    pos, vel = pos.float(), vel.float()
    order = torch.sort(_bucket(_cells(pos, _kernel_radius(d)), _buckets(pos.shape[0])), stable=True)[1]
    pos, vel = pos[order].contiguous(), vel[order].contiguous()
    scene = Scene(case["kind"], pos, d, case.get("delta_t", 0.05 * d), (0.0, 0.0, 0.0), box, boundary_pos=walls, fluid_vel=vel,
                  min_iters=limits[0], max_iters=limits[1])
    return scene, pos, vel


def _batch_scenes(case, seed):
    g, out = _generator(seed, 7), []
    u = np.random.RandomState(case["scenes"]).random_sample((case["scenes"], 4))  # sizes and kinds belong to the case
    d = case["spacing"]
    for k in range(case["scenes"]):
        n = int(round(math.exp(math.log(case["least"]) + u[k, 0] * math.log(case["most"] / case["least"]))))
        if u[k, 1] < 0.5:  # a dam-break column
            a, c = 0.5 + 1.5 * u[k, 2], 0.5 + 1.5 * u[k, 3]
            ny = max(2, int(round((n / (a * c)) ** (1.0 / 3.0))))
            nx, nz = max(2, int(round(a * ny))), max(2, int(round(c * ny)))
            pos = _block(nx, ny, nz, d, (0.0, 0.0, 0.0), case["jitter"], g)
            vel, box = _collapse(pos, 0.5 * u[k, 0], g), (2.5 * nx * d, 2.0 * ny * d, nz * d)
        else:  # a sphere on its way into a pool
            pos, vel, box = _drop(n, d, 0.5 * u[k, 2], case["jitter"], g)
        out.append(Scene("scene%d" % k, pos.float().cpu().numpy(), d, case["delta_t"], (0.0, 0.0, 0.0), box,
                         fluid_vel=vel.float().cpu().numpy()))
    return out


def _keys(case, seed):
    g = _generator(seed)
    n = case["count"]
    keys = torch.randint(0, 1 << case["bits"], (n,), generator=g, device=DEV, dtype=torch.int64)
    values = torch.randint(0, 1 << 31, (n,), generator=g, device=DEV, dtype=torch.int64)
    to32 = lambda v: torch.where(v >= 1 << 31, v - (1 << 32), v).to(torch.int32)  # noqa: E731
    return to32(keys), to32(values)


_stream = []


def _program_stream():
    """The one stream on which a program submits its work to the solver, contexts made one after another included."""
    if not _stream:
        _stream.append(torch.cuda.Stream())
    return _stream[0].cuda_stream


def prepare(case, seed):
    kind = case["kind"]
    if kind == "sort":
        keys, values = _keys(case, seed)
        return {"case": case, "sort": RadixSort(0), "keys": keys, "values": values, "k": torch.empty_like(keys),
                "v": torch.empty_like(values)}
    if kind == "batch":
        scenes = _batch_scenes(case, seed)
        torch.cuda.synchronize()
        batch = Batch(0, max_particles=sum(s.fluid_count for s in scenes), max_scenes=len(scenes), stream=_program_stream())
        ids = [batch.add_scene(s) for s in scenes]
        return {"case": case, "batch": batch, "ids": ids, "scenes": scenes}
    scene, pos, vel = _scene(case, seed)
    fluid = Fluid(0, _program_stream())
    torch.cuda.synchronize()
    setup_scene(fluid, scene)
    state = {"case": case, "fluid": fluid}
    if kind == "frame":
        eye = (3.0 * case["nx"] * case["spacing"], 2.0 * case["ny"] * case["spacing"], 4.0 * case["nz"] * case["spacing"])
        mid = (0.5 * case["nx"] * case["spacing"], 0.4 * case["ny"] * case["spacing"], 0.5 * case["nz"] * case["spacing"])
        state["camera"] = rendering.camera(eye, mid, fov_x_degrees=45.0)
        return state
    n = scene.fluid_count
    if case["memory"] == "host":
        pinned = [torch.empty((n, 3), dtype=torch.float32, pin_memory=True) for _ in range(4)]
        pinned[0].copy_(pos)
        pinned[1].copy_(vel)
        state["pinned"] = pinned
        state["pos"], state["vel"], state["out_pos"], state["out_vel"] = (t.numpy() for t in pinned)
    else:
        state["pos"], state["vel"] = pos, vel
        state["out_pos"], state["out_vel"] = torch.empty_like(pos), torch.empty_like(vel)
        state["out_rho"] = torch.empty(n, device=DEV, dtype=torch.float32)
    torch.cuda.synchronize()
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "sort":
        state["k"].copy_(state["keys"])
        state["v"].copy_(state["values"])
        state["sort"].enqueue(state["k"], state["v"], max_bits=case["bits"],
                              stream=torch.cuda.current_stream().cuda_stream)
        return state["k"], state["v"]
    if kind == "batch":
        batch = state["batch"]
        for sid, s in zip(state["ids"], state["scenes"]):
            batch.set_state(sid, s.fluid_pos, s.fluid_vel)
        batch.step(case["steps"])
        return [(batch.get_field(sid, "position", s.fluid_count), batch.get_field(sid, "velocity", s.fluid_count))
                for sid, s in zip(state["ids"], state["scenes"])]
    fluid = state["fluid"]
    if kind == "frame":
        return rendering.render(fluid, state["camera"], case["width"], case["height"])
    fluid.set_fluid_state(state["pos"], state["vel"])
    fluid.step(case["steps"])
    fluid.get_fluid_state(state["out_pos"], state["out_vel"])
    if case["memory"] == "host":
        return state["out_pos"], state["out_vel"]
    fluid.get_field("density", out=state["out_rho"])
    return state["out_pos"], state["out_vel"], state["out_rho"]


# ------------------------------------------------------------------------------------------------ work


def _particles(case):
    if case["kind"] in ("drop", "batch"):
        if case["kind"] == "drop":
            return case["count"]
        lo, hi = case["least"], case["most"]
        return int(case["scenes"] * (hi - lo) / math.log(hi / lo))
    return case["nx"] * case["ny"] * case["nz"] * (2 if case["kind"] == "blocks" else 1)


def work(case):
    if case["kind"] == "sort":
        return {"bytes": 16 * case["count"], "flops": 0}
    n = _particles(case)
    if case["kind"] == "frame":
        return {"bytes": 16 * n + 3 * case["width"] * case["height"], "flops": 40 * n}
    # state in and out once per pass (and the density, where it is taken); per step 33 neighbours within the kernel
    # radius of each particle: density 11, normal 14 and forces 60 operations a pair, each corrective iteration 11 + 20
    pairs = 33 * n * case["steps"]
    return {"bytes": 52 * n, "flops": pairs * (85 + 31 * case["iterations"])}


# ----------------------------------------------------------------------------------------------- exact


class _Near:
    """The pairs of the 27-bucket walk around targets (float32 positions) over sources sorted by bucket; a bucket that two of
    the 27 cells share is visited twice. Only pairs closer than `reach` are kept."""

    def __init__(self, targets, sources, keys, buckets, h, reach):
        first = torch.searchsorted(keys, torch.arange(buckets + 1, device=DEV))
        c, self.parts = _cells(targets, h), []
        for o in range(27):
            off = torch.tensor([o % 3 - 1, o // 3 % 3 - 1, o // 9 - 1], device=DEV)
            b = _bucket(c + off, buckets)
            start, count = first[b], first[b + 1] - first[b]
            i = torch.repeat_interleave(torch.arange(targets.shape[0], device=DEV), count)
            j = torch.arange(i.shape[0], device=DEV) - torch.repeat_interleave(torch.cumsum(count, 0) - count, count) + start[i]
            near = (targets[i] - sources[j]).square().sum(1) <= reach * reach
            self.parts.append((i[near].to(torch.int32), j[near].to(torch.int32)))

    def sum(self, like, term):
        out = torch.zeros_like(like)
        for i, j in self.parts:
            out.index_add_(0, i, term(i, j))
        return out


def _poly6(r2, h2):
    return torch.where(r2 > h2, 0.0, h2 - r2).pow(3)


def exact(case, seed):
    if case["kind"] == "sort":
        keys, values = _keys(case, seed)
        k, order = torch.sort(keys.to(torch.int64) & 0xFFFFFFFF, stable=True)
        return torch.where(k >= 1 << 31, k - (1 << 32), k).to(torch.int32), values[order]
    if case["kind"] in ("batch", "frame", "blocks") or case["steps"] > 1:
        return None  # many steps of a chaotic system, an image of bytes, or too many particles
    scene, pos, vel = _scene(case, seed)
    h = _kernel_radius(case["spacing"])
    h2, d, rho0, g = _f32(h * h), 0.5 * h, 1000.0, _f32(-9.81)
    mass, dt, tension = _f32(rho0 * d ** 3), _f32(case["delta_t"]), 0.5
    visc = _f32(scene.viscosity_constant())
    k6, k6d = 315.0 / (64.0 * math.pi * h ** 9), -945.0 / (32.0 * math.pi * h ** 9)
    kv, ks, kt = 45.0 / (math.pi * h ** 6), -45.0 / (math.pi * h ** 6), 32.0 / (math.pi * h ** 9)
    grid = torch.arange(-3, 4, dtype=torch.float64) * d
    at = torch.stack(torch.meshgrid(grid, grid, grid, indexing="ij"), -1).reshape(-1, 3)
    r2 = at.square().sum(1)
    grad = torch.where((r2 < h2 * (1 - 1e-9))[:, None], -k6d * (h2 - r2).square()[:, None] * at, 0.0)
    beta = dt * dt * mass * mass * 2.0 / (rho0 * rho0)
    delta = float(1.0 / (beta * (grad.sum(0).square().sum() + grad.square().sum())))

    n = pos.shape[0]
    buckets = _buckets(n)
    key, order = torch.sort(_bucket(_cells(pos, h), buckets), stable=True)
    x32 = pos[order]
    x, v = x32.double(), vel[order].double()
    reach = 1.6 * h
    near = _Near(x32, x32, key, buckets, h, reach)
    wall = near_wall = wall_near = None
    if scene.boundary_count:
        b32 = scene.boundary_pos
        bkey, border = torch.sort(_bucket(_cells(b32, h), buckets), stable=True)
        b32 = b32[border]
        wall = b32.double()
        near_wall, wall_near = _Near(x32, b32, bkey, buckets, h, reach), _Near(b32, x32, key, buckets, h, reach)

    def dist2(a, b, i, j):
        return (a[i] - b[j]).square().sum(1)

    rho = near.sum(x[:, 0], lambda i, j: _poly6(dist2(x, x, i, j), h2))
    if wall is not None:
        rho += near_wall.sum(x[:, 0], lambda i, j: _poly6(dist2(x, wall, i, j), h2))
    rho *= mass * k6
    normal = near.sum(x, lambda i, j: (x[i] - x[j]) * ((h2 - dist2(x, x, i, j)).clamp_min(0).square() / rho[j])[:, None])
    normal *= h * mass * k6d

    def viscous(i, j):
        r = dist2(x, x, i, j).sqrt()
        return (v[j] - v[i]) * ((h - r).clamp_min(0) / rho[j])[:, None]

    def surface(i, j):
        e = x[i] - x[j]
        r = e.square().sum(1).sqrt()
        on = (r > _f32(1e-4)) & (r < h)
        t = (h - r).pow(3) * r.pow(3)
        w = torch.where(r <= 0.5 * h, 2.0 * t - h ** 6 / 64.0, t)
        f = (w / r.clamp_min(1e-12))[:, None] * e * (tension * mass * mass * kt) + (normal[i] - normal[j]) * (tension * mass)
        return torch.where(on, 2.0 * rho0 / (rho[i] + rho[j]), 0.0)[:, None] * -f

    other = near.sum(x, viscous) * (visc * mass * kv) + near.sum(x, surface)
    other[:, 1] += mass * g
    push, press = torch.zeros_like(x), torch.zeros_like(rho)
    wall_press = None if wall is None else torch.zeros_like(wall[:, 0])
    for it in range(1, scene.max_iters + 1):
        xs = x + (v + (other + push) / mass * dt) * dt
        if wall is not None:
            at_wall = wall_near.sum(wall_press, lambda i, j: _poly6(dist2(wall, xs, i, j), h2)) * (mass * k6)
            wall_press = wall_press + delta * (at_wall - rho0).clamp_min(0)
        rs = near.sum(rho, lambda i, j: _poly6(dist2(xs, xs, i, j), h2))
        if wall is not None:
            rs += near_wall.sum(rho, lambda i, j: _poly6(dist2(xs, wall, i, j), h2))
        error = (rs * (mass * k6) - rho0).clamp_min(0)
        press = press + delta * error
        q = press / rho.square()

        def spiky(e, s):
            r = e.square().sum(1).sqrt()
            on = (r <= h) & (r >= 1e-4)
            return e * torch.where(on, (h - r).square() / r.clamp_min(1e-12) * s, 0.0)[:, None]

        push = near.sum(x, lambda i, j: spiky(x[i] - x[j], q[i] + q[j]))
        if wall is not None:
            qw = wall_press / (rho0 * rho0)
            push += near_wall.sum(x, lambda i, j: spiky(x[i] - wall[j], q[i] + qw[j]))
        push *= -ks * mass * mass
        if it >= scene.min_iters and float(error.max()) / rho0 < scene.threshold:
            break
    v = v + (other + push) / mass * dt
    x = x + v * dt
    hi = torch.tensor([_f32(b) for b in scene.box_hi], device=DEV, dtype=torch.float64)
    below, above = x < 0, x > hi
    x = torch.minimum(x.clamp_min(0), hi)
    v = torch.where((below & (v < 0)) | (above & (v > 0)), -scene.restitution * v, v)
    return (x, v) if case["memory"] == "host" else (x, v, rho)
