"""The work that users have the framework do, as a list of timed cases.

Every case goes through the public Python entry points (which are thin calls
of the C interface): the fused update, the reference-named stage calls, the
unified-memory step with a distance-map obstacle, batches of scenes, the
neural SDF's inference and training, and the distance map of a mesh.  Steps
change the particle state in place, so a pass first puts the start state back
(one device copy), as parameter sweeps and optimisers that restart from a
snapshot do; every pass then does the same work.

``exact`` restates the same mathematics in float64 with torch.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from fullc0ntact_gb300 import dem, scenes, sdf
from fullc0ntact_gb300.params import make_params

DEV = "cuda"
R_MED, R_SIGMA, R_MAX = 1.0 / 512.0, 0.25, 2.0 / 512.0  # the polydisperse scenes' radii
MARGIN = 0.05        # margin of every distance map around its obstacle
NUM_SHAPES = 8       # obstacles of the batched scenes
ADAM = (0.9, 0.999, 1e-8)


def listed() -> list:
    return [
        # an interactive host stepping a small scene one update per call: launches and host time
        dict(name="step_2k", kind="update", scene="lattice", n=2000, grid=64, steps=1),
        # the reference demo's scene (16,384 spheres, 64^3 cells), 20 updates between two outputs
        dict(name="lattice_16k", kind="update", scene="lattice", n=16384, grid=64, steps=20),
        # the headline scene at full size: lognormal radii, 30% volume fraction, 256^3 cells
        dict(name="gas_4m", kind="update", scene="gas", n=4194304, grid=256, steps=4),
        # the same spheres once gravity has settled them: crowded cells at the floor
        dict(name="pile_1m", kind="update", scene="pile", n=1000003, grid=256, steps=3),
        # drop-in host code: the five reference-named calls of one update, polydisperse, ragged size
        dict(name="stages_100k", kind="stages", scene="gas", n=100003, grid=128),
        # the same calls on a million equal spheres
        dict(name="stages_1m", kind="stages", scene="fall", n=1048576, grid=256),
        # spheres falling onto a torus given as a distance map, unified-memory step with forces
        dict(name="torus_1m", kind="um", n=1048576, grid=256, steps=5, net=False),
        # many independent box scenes of uneven size in one batch, replayed from a graph
        dict(name="batch_boxes", kind="batch", obstacles="none", num=128, lo=1024, hi=65536,
             steps=10),
        # scenes over eight obstacles, the map query culled by the shape-conditioned network
        dict(name="batch_obstacles", kind="batch", obstacles="net", num=40, lo=4096, hi=131072,
             steps=6),
        # distances of a million points from the trained network (tensor-core inference)
        dict(name="infer_1m", kind="infer", n=1048576, inputs=3, hidden=64, layers=3),
        # one epoch of training the obstacle network: mini-batches of 2,048 samples
        dict(name="train_64k", kind="train", n=65536, batch=2048, inputs=3, hidden=64, layers=3),
        # obstacle set-up: the 128-cell distance map of a 256 x 64-quad torus mesh
        dict(name="mesh_map", kind="mesh", nu=256, nv=64, cells=128),
    ]


def _spread(rng, lo: int, hi: int) -> int:
    """A whole number log-uniform in [lo, hi]."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng) -> dict:
    kind = rng.choice(["update", "update", "update", "stages", "stages", "um", "um", "batch",
                       "batch", "infer", "train", "mesh"])
    if kind in ("update", "stages"):
        scene = rng.choice(["lattice", "gas", "pile", "fall"] if kind == "update"
                           else ["gas", "fall"])
        n = _spread(rng, *dict(lattice=(1000, 200000), gas=(4000, 4194304),
                               pile=(50000, 1000003), fall=(20000, 1048576))[scene])
        grid = 64 if scene == "lattice" else 256 if scene == "pile" or n > 200000 else 128
        case = dict(kind=kind, scene=scene, n=n, grid=grid)
        if kind == "update":
            case["steps"] = max(1, min(_spread(rng, 1, 32), 16000000 // n,
                                       3 if scene == "pile" else 32))
        return case
    if kind == "um":
        n = _spread(rng, 20000, 1048576)
        return dict(kind="um", n=n, grid=256, steps=rng.randint(1, 6), net=rng.random() < 0.4)
    if kind == "batch":
        obstacles = rng.choice(["none", "exact", "net"])
        if obstacles == "none":
            return dict(kind="batch", obstacles="none", num=rng.randint(3, 128), lo=1024,
                        hi=_spread(rng, 4096, 65536), steps=rng.randint(1, 10))
        return dict(kind="batch", obstacles=obstacles, num=rng.randint(2, 40), lo=4096,
                    hi=_spread(rng, 16384, 131072), steps=rng.randint(1, 6))
    hidden, layers = rng.choice([(64, 2), (64, 3), (128, 2), (128, 3)])
    inputs = rng.choice([3, 3 + NUM_SHAPES])
    if kind == "infer":
        return dict(kind="infer", n=_spread(rng, 1000, 2000000), inputs=inputs, hidden=hidden,
                    layers=layers)
    if kind == "train":
        return dict(kind="train", n=_spread(rng, 16384, 131072),
                    batch=rng.choice([1024, 2048, 4096, 8192]), inputs=inputs, hidden=hidden,
                    layers=layers)
    return dict(kind="mesh", nu=_spread(rng, 24, 256), nv=_spread(rng, 12, 64),
                cells=rng.randint(24, 128))


# --- inputs ------------------------------------------------------------------

def _radii(rng, n: int) -> np.ndarray:
    r = R_MED * np.exp(R_SIGMA * rng.standard_normal(n))
    return np.minimum(r, R_MAX).astype(np.float32)


def _scene(case: dict, seed: int) -> dict:
    """One scene dict (pos, vel, params ...) of a single-scene case."""
    n, grid, name = case["n"], case["grid"], case.get("scene", "fall")
    if name == "lattice":
        return scenes.lattice_scene(n, seed)
    if name == "fall":
        return scenes.torus_fall_scene(n, seed, grid)
    rng = np.random.default_rng(seed)
    pos, vel = np.zeros((n, 4), np.float32), np.zeros((n, 4), np.float32)
    pos[:, 3] = _radii(rng, n)
    vel[:, :3] = rng.uniform(-0.01, 0.01, (n, 3))
    if name == "gas":  # the packed scene after its first step: uniform, 30% volume fraction
        side = (n * scenes.lognormal_mean_volume(R_MED, R_SIGMA) / 0.30) ** (1.0 / 3.0)
        side = min(side, 2.0 - 4.0 * R_MAX)
        pos[:, :3] = rng.uniform(-side / 2, side / 2, (n, 3))
    else:  # pile: 24 spheres per floor cell, thinning by 1/e every 3 cells
        cell = 2.0 * R_MAX
        side = min(cell * math.sqrt(n / 72.0), 1.98)
        pos[:, :2] = rng.uniform(-side / 2, side / 2, (n, 2))
        pos[:, 2] = -1.0 + pos[:, 3] + np.minimum(rng.exponential(3.0 * cell, n), 1.0)
        vel *= 0.1
    params = make_params(n, (grid,) * 3, particle_radius=R_MAX, cell_size=2.0 * R_MAX)
    return dict(pos=pos, vel=vel, params=params, radius_from_w=True, dt=0.5)


def _batch_scenes(case: dict, seed: int):
    """(scene dicts, obstacles, obstacle of each scene) of a batch case."""
    rng = np.random.default_rng(seed)
    sizes = np.exp(np.linspace(math.log(case["lo"]), math.log(case["hi"]), case["num"]))
    sizes = rng.permutation(sizes.astype(np.int64) + np.arange(case["num"]) * 7 % 17)
    if case["obstacles"] != "none":
        obs = scenes.obstacle_set(NUM_SHAPES)
        shape = [k % NUM_SHAPES for k in range(case["num"])]
        return [scenes.obstacle_scene(int(n), obs[s], int(rng.integers(1 << 30)))
                for n, s in zip(sizes, shape)], obs, shape
    out = []
    for n in sizes:  # radii U[1/512, 1/256], 25% volume fraction, the cube is the scene's box
        n = int(n)
        pos, vel = np.zeros((n, 4), np.float32), np.zeros((n, 4), np.float32)
        r = rng.uniform(R_MED, R_MAX, n).astype(np.float32)
        side = (float((4.0 / 3.0 * np.pi * r.astype(np.float64) ** 3).sum()) / 0.25) ** (1 / 3)
        half = np.float32(side / 2)
        pos[:, :3] = rng.uniform(-1.0, 1.0, (n, 3)) * (half - r[:, None])
        pos[:, 3] = r
        vel[:, :3] = rng.uniform(-0.01, 0.01, (n, 3))
        g = 4
        while g * 2 * R_MAX < side:
            g *= 2
        params = make_params(n, (g,) * 3, R_MAX, 2.0 * R_MAX, (-float(half),) * 3,
                             collider_pos=(10.0,) * 3, collider_radius=0.0)
        out.append(dict(pos=pos, vel=vel, params=params, radius_from_w=True, dt=0.5,
                        box_lo=np.full(3, -half), box_hi=np.full(3, half)))
    return out, [], []


@functools.lru_cache(maxsize=None)
def _torus_net():
    """The torus map with its trained network and culling threshold, as a user keeps them."""
    dmap = dem.DistanceMap.torus(0.3, 0.1, 128, MARGIN)
    net = sdf.SdfNet(3, 64, 3, seed=5)
    net.normalize_to(dmap)
    net.train(sdf.samples(dmap, 800000, 0.6, 0.05, seed=21), epochs=10, batch=2048, lr=5e-3,
              band=0.02)
    skin, _ = sdf.calibrate_skin(net, [dmap], 1.0 / 256.0, shaped=False)
    return dmap, net, skin


@functools.lru_cache(maxsize=None)
def _shape_net():
    """The obstacle set's maps, the shape-conditioned network and its culling threshold."""
    maps = sdf.obstacle_maps(scenes.obstacle_set(NUM_SHAPES), 128, MARGIN)
    net, _ = sdf.shape_net(maps, samples_per_map=200000, epochs=10)
    skin, _ = sdf.calibrate_skin(net, maps, R_MAX)
    return maps, net, skin


def _points(case: dict, seed: int):
    """Points in the network's box with the distance to a torus, and shape codes."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    p = torch.rand(case["n"], 4, generator=g, device=DEV) * 0.9 - 0.45
    rho = p[:, :2].norm(dim=1) - 0.3
    p[:, 3] = (rho * rho + p[:, 2] * p[:, 2]).sqrt() - 0.1
    codes = None
    if case["inputs"] > 3:
        codes = torch.randint(case["inputs"] - 3, (case["n"],), generator=g, device=DEV,
                              dtype=torch.int32)
    return p, codes


def _weights(case: dict, seed: int) -> np.ndarray:
    """FP32 parameters at the usual initial scale, biases included."""
    rng = np.random.default_rng(seed)
    d, h = case["inputs"], case["hidden"]
    parts = [rng.uniform(-1, 1, h * d) * math.sqrt(2.0), rng.uniform(-0.5, 0.5, h)]
    for _ in range(case["layers"] - 1):
        parts += [rng.uniform(-1, 1, h * h) * math.sqrt(6.0 / h), rng.uniform(-0.5, 0.5, h)]
    parts += [rng.uniform(-1, 1, h) * math.sqrt(6.0 / h), rng.uniform(-0.1, 0.1, 1)]
    return np.concatenate(parts).astype(np.float32)


def _mesh(case: dict, seed: int):
    """A torus mesh with ripples that depend on the seed, in the box of the plain torus."""
    rng = np.random.default_rng(seed)
    verts, tris = scenes.torus_mesh(0.3, rng.uniform(0.07, 0.12), case["nu"], case["nv"])
    u = np.arctan2(verts[:, 1], verts[:, 0])
    verts = verts * (1.0 + 0.03 * np.sin(rng.integers(2, 6) * u + rng.uniform(0, 6)))[:, None]
    lo, hi = verts.min(axis=0), verts.max(axis=0)
    half = np.array([0.4, 0.4, 0.1])
    verts = np.clip((verts - lo) / (hi - lo) * (2 * half) - half, -half, half)
    return verts.astype(np.float32), tris


def _restartable(owner, pos: torch.Tensor, vel: torch.Tensor) -> torch.Tensor:
    """Gives `owner` one buffer for pos and vel; returns the start state to copy into it."""
    start = torch.stack([pos, vel])
    owner.state = start.clone()
    owner.pos, owner.vel = owner.state[0], owner.state[1]
    return start


def prepare(case: dict, seed: int):
    kind = case["kind"]
    if kind in ("update", "stages"):
        ds = dem.DeviceScene(_scene(case, seed), DEV)
        return case, ds, _restartable(ds, ds.pos, ds.vel)
    if kind == "um":
        if case["net"]:
            dmap, net, skin = _torus_net()
            kw = dict(net=net, skin=skin)
        else:
            dmap, kw = dem.DistanceMap.torus(0.3, 0.1, 128, MARGIN), {}
        us = dem.UmScene(_scene(case, seed), dmap, DEV)
        return case, us, _restartable(us, us.pos, us.vel), kw
    if kind == "batch":
        scs, obs, shape = _batch_scenes(case, seed)
        b = dem.Batch(scs, DEV)
        if case["obstacles"] == "exact":
            b.set_obstacles(sdf.obstacle_maps(obs, 128, MARGIN), shape)
        elif case["obstacles"] == "net":
            maps, net, skin = _shape_net()
            b.set_obstacles(maps, shape, net, skin)
        return case, b, _restartable(b, b.pos, b.vel)
    if kind in ("infer", "train"):
        net = sdf.SdfNet(case["inputs"], case["hidden"], case["layers"], seed=1)
        net.set_normalization([0.0] * 3, [1.0 / 0.45] * 3, 0.45)
        weights = _weights(case, seed)
        net.set_params(weights)
        return case, net, _points(case, seed), weights
    return case, _mesh(case, seed)


def run(state):
    case, kind = state[0], state[0]["kind"]
    if kind in ("update", "stages"):
        _, ds, start = state
        ds.state.copy_(start)
        if kind == "update":
            ds.update(case["steps"])
        else:
            ds.stages()
        return dict(pos=ds.pos, vel=ds.vel, sorted_pos=ds.sorted_pos, sorted_vel=ds.sorted_vel,
                    hash=ds.hash, index=ds.index, cell_start=ds.cell_start)
    if kind == "um":
        _, us, start, kw = state
        us.state.copy_(start)
        us.update(case["steps"], **kw)
        return dict(pos=us.pos, vel=us.vel, force=us.force, hash=us.hash, index=us.index,
                    cell_start=us.cell_start)
    if kind == "batch":
        _, b, start = state
        b.state.copy_(start)
        b.update(case["steps"], graph=True)
        return dict(pos=b.pos, vel=b.vel)
    if kind == "infer":
        _, net, (pts, codes), _ = state
        return net.infer(pts, codes)
    if kind == "train":
        _, net, (pts, codes), weights = state
        net.set_params(weights)
        loss = net.train(pts, codes, epochs=1, batch=case["batch"], lr=1e-3, band=0.02)
        return dict(loss=loss, params=net.get_params())
    _, (verts, tris) = state
    return dem.DistanceMap.from_mesh(verts, tris, case["cells"], MARGIN).vertices()


def _batch_size(case: dict) -> float:
    """Particles of a batch case (mean of a log-uniform size)."""
    lo, hi = case["lo"], case["hi"]
    return case["num"] * (hi - lo) / math.log(hi / lo)


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind in ("update", "stages", "um", "batch"):
        n = _batch_size(case) if kind == "batch" else case["n"]
        cells = 0 if kind == "batch" else case["grid"] ** 3
        steps = case.get("steps", 1)
        # in: pos, vel; out: pos, vel and, where the call gives them, the sorted
        # copies, hash, index (and force) and the cell table
        out = 32 if kind == "batch" else 32 + 32 + 8 + (12 if kind == "um" else 0)
        # per particle and step: the pairs in contact (about 2.4 in the gas,
        # 30 in the pile, 1 elsewhere) at 60 operations and the integration
        touching = dict(gas=2.4, pile=30.0).get(case.get("scene"), 1.0)
        return dict(bytes=float(n * (32 + out) + 4 * cells),
                    flops=float(n * steps * (60 * touching + 30)))
    if kind in ("infer", "train"):
        d, h, layers, n = case["inputs"], case["hidden"], case["layers"], case["n"]
        macs = h * d + (layers - 1) * h * h + h
        params = macs + layers * h + 1
        code = 4 if d > 3 else 0
        if kind == "infer":
            return dict(bytes=float(n * (16 + code + 4) + 4 * params), flops=2.0 * n * macs)
        return dict(bytes=float(n * (16 + code) + 8 * params), flops=6.0 * n * macs)
    side = case["cells"] + 1
    verts = side * side * max(2, int(side * 0.4))
    tris = 2 * case["nu"] * case["nv"]
    # each vertex: at least one closest-point evaluation and its output
    return dict(bytes=float(16 * verts + 12 * (tris // 2) + 12 * tris), flops=100.0 * verts)


# --- the same in float64 -----------------------------------------------------

def _t(a) -> torch.Tensor:
    return torch.as_tensor(np.asarray(a), device=DEV).double()


class _World:
    """The scenes of a case side by side in float64: state, radii, cells, box, obstacle."""

    def __init__(self, scene_list: list):
        p = scene_list[0]["params"]
        sizes = torch.tensor([s["pos"].shape[0] for s in scene_list], device=DEV)

        def each(rows, dtype=torch.float64):
            return torch.repeat_interleave(torch.tensor(rows, dtype=dtype, device=DEV), sizes, 0)
        par = [s["params"] for s in scene_list]
        pos = _t(np.concatenate([s["pos"] for s in scene_list]))
        self.x, self.w = pos[:, :3].contiguous(), pos[:, 3]
        vel = _t(np.concatenate([s["vel"] for s in scene_list]))
        self.v, self.vw = vel[:, :3].contiguous(), vel[:, 3]
        poly = scene_list[0]["radius_from_w"]
        self.r = self.w if poly else torch.full_like(self.w, p.particleRadius)
        self.origin = each([list(q.worldOrigin) for q in par])
        self.cell = each([[q.cellSize[0]] for q in par])
        self.grid = each([list(q.gridSize) for q in par], torch.int64)
        cells = np.cumsum([0] + [int(np.prod(list(q.gridSize))) for q in par])
        self.base, self.cells = each(cells[:-1].tolist(), torch.int64), int(cells[-1])
        self.lo = each([[float(c) for c in s.get("box_lo", (-1.0,) * 3)] for s in scene_list])
        self.hi = each([[float(c) for c in s.get("box_hi", (1.0,) * 3)] for s in scene_list])
        self.p, self.dt, self.sizes = p, scene_list[0]["dt"], sizes
        self.gravity = _t(list(p.gravity))

    def key(self, c: torch.Tensor) -> torch.Tensor:
        c = c & (self.grid - 1)
        return self.base + (c[:, 2] * self.grid[:, 1] + c[:, 1]) * self.grid[:, 0] + c[:, 0]

    def term(self, rel, dist, cd, rv, attraction):
        nrm = rel / dist[:, None]
        tan = rv - (rv * nrm).sum(1, keepdim=True) * nrm
        return (-self.p.spring * (cd - dist)[:, None] * nrm + self.p.damping * rv
                + self.p.shear * tan + attraction * rel)

    def forces(self, collider: bool) -> torch.Tensor:
        c = torch.floor((self.x - self.origin) / self.cell).long()
        h = self.key(c)
        order = torch.argsort(h)
        count = torch.bincount(h, minlength=self.cells)
        first = torch.cumsum(count, 0) - count
        force = torch.zeros_like(self.x)
        for k in range(27):
            off = torch.tensor([k % 3 - 1, k // 3 % 3 - 1, k // 9 - 1], device=DEV)
            nk = self.key(c + off)
            a, m = first[nk], count[nk]
            live = torch.nonzero(m > 0)[:, 0]
            q = 0
            while live.numel():
                j = order[a[live] + q]
                d2 = (self.x[j] - self.x[live]).square().sum(1)
                hit = (d2 < (self.r[live] + self.r[j]).square()) & (j != live)
                i, j = live[hit], j[hit]
                rel = self.x[j] - self.x[i]
                force.index_add_(0, i, self.term(rel, rel.norm(dim=1), self.r[i] + self.r[j],
                                                 self.v[j] - self.v[i], self.p.attraction))
                q += 1
                live = live[m[live] > q]
        if collider:
            rel = _t(list(self.p.colliderPos)) - self.x
            dist, cd = rel.norm(dim=1), self.r + self.p.colliderRadius
            i = torch.nonzero(dist < cd)[:, 0]
            force.index_add_(0, i, self.term(rel[i], dist[i], cd[i], -self.v[i], 0.0))
        return force

    def advance(self) -> None:
        self.v = (self.v + self.gravity * self.dt) * self.p.globalDamping
        self.x = self.x + self.v * self.dt

    def face(self, axes, bound, above: bool) -> None:
        """Clamps the axes to the faces of a box and damps the velocity there."""
        for a in axes:
            lim = bound[:, a] - self.r if above else bound[:, a] + self.r
            out = self.x[:, a] > lim if above else self.x[:, a] < lim
            self.x[:, a] = torch.where(out, lim, self.x[:, a])
            self.v[:, a] = torch.where(out, self.v[:, a] * self.p.boundaryDamping, self.v[:, a])

    def box(self) -> None:
        self.face(range(3), self.hi, True)
        self.face(range(3), self.lo, False)

    def touch(self, field: "_Field", rows: torch.Tensor) -> None:
        """The distance-map contact of the particles `rows`."""
        dist, cp, inside = field(self.x[rows])
        i = rows[inside & (dist < self.r[rows])]
        hit = inside & (dist < self.r[rows])
        n = self.x[i] - cp[hit]
        n = n / n.norm(dim=1, keepdim=True)
        self.x[i] += n * (self.r[i] - dist[hit] + 0.1 * self.r[i])[:, None]
        bd = self.p.boundaryDamping
        self.v[i] *= _t([0.5 * bd, 0.5 * bd, 0.7 * bd])


class _Field:
    """Trilinear distance map of a torus or rounded box, vertices rounded to float32."""

    def __init__(self, ob: dict, cells: int = 128):
        f = np.float32
        if ob["kind"] == "torus":
            big, tube = f(ob["R"]), f(ob["r"])
            ext = [f(big + tube + f(MARGIN))] * 2 + [f(tube + f(MARGIN))]
        else:
            half = [f(h) for h in ob["h"]]
            ext = [f(h + f(MARGIN)) for h in half]
        self.cs = f(f(2) * max(ext)) / f(cells)
        num = [int(math.ceil(f(f(2) * e) / self.cs)) for e in ext]
        if ob["kind"] == "torus":
            num[:2] = [cells, cells]
            vmin = [-ext[0], -ext[1], f(-0.5) * f(num[2]) * self.cs]
        else:
            vmin = [f(-0.5) * f(c) * self.cs for c in num]
        axes = [vmin[a] + np.arange(num[a] + 1, dtype=f) * self.cs for a in range(3)]
        z, y, x = torch.meshgrid(*[_t(axes[a]) for a in (2, 1, 0)], indexing="ij")
        p = torch.stack([x, y, z], -1).reshape(-1, 3)
        if ob["kind"] == "torus":
            ring = p.clone()
            ring[:, 2] = 0
            ring = ring / ring.norm(dim=1, keepdim=True).clamp_min(1e-300) * float(big)
            away = p - ring
            o = away.norm(dim=1, keepdim=True)
            d, cp = o[:, 0] - float(tube), ring + away / o.clamp_min(1e-300) * float(tube)
        else:
            rr = float(f(ob["rounding"]))
            inner = _t(half) - rr
            near = torch.minimum(torch.maximum(p, -inner), inner)
            o = (p - near).norm(dim=1, keepdim=True)
            depth, axis = (p.abs() - inner).max(dim=1)
            flat = p.clone()
            flat.scatter_(1, axis[:, None],
                          torch.where(p.gather(1, axis[:, None]) < 0, -1.0, 1.0)
                          * (inner + rr)[axis][:, None])
            out = o[:, 0] > 0
            d = torch.where(out, o[:, 0], depth) - rr
            cp = torch.where(out[:, None], near + rr * (p - near) / o.clamp_min(1e-300), flat)
        self.val = torch.cat([d[:, None], cp], 1).float().double()
        self.num, self.vmin = torch.tensor(num, device=DEV), _t(vmin)
        self.vmax = _t([vmin[a] + f(num[a]) * self.cs for a in range(3)])

    def __call__(self, q: torch.Tensor):
        inside = ((q >= self.vmin) & (q <= self.vmax)).all(1)
        s = (q - self.vmin) / float(self.cs)
        i = torch.minimum(s.long().clamp_min(0), self.num - 1)
        w = s - i
        nx, ny = (self.num[:2] + 1).tolist()
        val = torch.zeros(q.shape[0], 4, dtype=torch.float64, device=DEV)
        for k in range(8):
            b = torch.tensor([k & 1, k >> 1 & 1, k >> 2], device=DEV)
            wt = torch.where(b > 0, w, 1 - w).prod(1)
            c = i + b
            at = ((c[:, 2] * ny + c[:, 1]) * nx + c[:, 0]).clamp(0, self.val.shape[0] - 1)
            val += wt[:, None] * self.val[at]
        return val[:, 0], val[:, 1:], inside


def _exact_um(case: dict, seed: int) -> dict:
    w = _World([_scene(case, seed)])
    field = _Field(dict(kind="torus", R=0.3, r=0.1))
    rows = torch.arange(w.x.shape[0], device=DEV)
    planes = torch.zeros_like(w.x)
    for _ in range(case["steps"]):
        force = w.forces(False)
        w.v = w.v + force
        w.advance()
        flat = w.x.clone()
        flat[:, 2] = 0
        length = flat.norm(dim=1, keepdim=True)
        w.touch(field, rows)
        out = length > 1.0  # the cylinder of radius 1 around z
        away = flat / length.clamp_min(1e-300) * (length - 1.0 + w.r[:, None])
        w.x = torch.where(out, w.x - away, w.x)
        w.v[:, :2] = torch.where(out, w.v[:, :2] * w.p.boundaryDamping, w.v[:, :2])
        w.face([2], planes + 10.0, True)
        w.face([2], planes - 1.0, False)
    return dict(pos=torch.cat([w.x, w.w[:, None]], 1), vel=torch.cat([w.v, w.w[:, None]], 1),
                force=force, hash=None, index=None, cell_start=None)


def _exact_scenes(case: dict, seed: int) -> dict:
    """Fused updates, stage calls and batches: integrate in the box, then collide."""
    fields, rows = [], []
    if case["kind"] == "batch":
        scs, obs, shape = _batch_scenes(case, seed)
        w = _World(scs)
        if obs:
            of = torch.repeat_interleave(torch.tensor(shape, device=DEV), w.sizes)
            fields = [_Field(ob) for ob in obs]
            rows = [torch.nonzero(of == k)[:, 0] for k in range(len(obs))]
    else:
        w = _World([_scene(case, seed)])
    for _ in range(case.get("steps", 1)):
        w.advance()
        for f, at in zip(fields, rows):
            w.touch(f, at)
        w.box()
        w.v = w.v + w.forces(case["kind"] != "batch")
    out = dict(pos=torch.cat([w.x, w.w[:, None]], 1),
               vel=torch.cat([w.v, torch.zeros_like(w.w)[:, None]], 1))
    if case["kind"] != "batch":  # the sorted copies follow the cells of the rounded positions
        out.update(sorted_pos=None, sorted_vel=None, hash=None, index=None, cell_start=None)
    return out


def _forward(case: dict, params: torch.Tensor, pts: torch.Tensor, codes) -> torch.Tensor:
    """The network's output in units of its output scale."""
    d, h = case["inputs"], case["hidden"]
    x = pts[:, :3].double() * float(np.float32(1.0 / 0.45))
    if d > 3:
        x = torch.cat([x, torch.nn.functional.one_hot(codes.long(), d - 3).double()], 1)
    at = 0
    for k in [d] + [h] * (case["layers"] - 1):
        x = torch.nn.functional.silu(x @ params[at:at + h * k].view(h, k).T
                                     + params[at + h * k:at + h * k + h])
        at += h * k + h
    return x @ params[at:at + h] + params[at + h]


def _exact_train(case: dict, seed: int) -> dict:
    pts, codes = _points(case, seed)
    p = _t(_weights(case, seed)).requires_grad_()
    m, v = torch.zeros_like(p), torch.zeros_like(p)
    batches = -(-case["n"] // case["batch"])
    b1, b2, eps = ADAM
    total = 0.0
    for b in range(batches):
        part = slice(b * case["batch"], min(case["n"], (b + 1) * case["batch"]))
        dist = pts[part, 3].double()
        y = _forward(case, p, pts[part], None if codes is None else codes[part])
        weight = torch.where(dist.abs() < float(np.float32(0.02)), 10.0, 1.0)
        loss = (weight * (y - dist / float(np.float32(0.45))).square()).mean()
        g, = torch.autograd.grad(loss, p)
        lr = 1e-3 * (0.05 + 0.95 * 0.5 * (1.0 + math.cos(math.pi * b / batches)))
        with torch.no_grad():
            m = b1 * m + (1 - b1) * g
            v = b2 * v + (1 - b2) * g * g
            p -= lr * (m / (1 - b1 ** (b + 1))) / ((v / (1 - b2 ** (b + 1))).sqrt() + eps)
        total += float(loss)
    return dict(loss=total / batches, params=p.detach())


def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind in ("update", "stages", "batch"):
        return _exact_scenes(case, seed)
    if kind == "um":
        return _exact_um(case, seed)
    if kind == "infer":
        pts, codes = _points(case, seed)
        p = _t(_weights(case, seed))
        with torch.no_grad():
            return _forward(case, p, pts, codes) * float(np.float32(0.45))
    if kind == "train":
        return _exact_train(case, seed)
    return None  # every vertex against every triangle in 64 bits takes minutes
