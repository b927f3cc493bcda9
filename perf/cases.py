"""The work a user of this framework has it do, as cases that a timing program can run.

Each case goes through the package's public entry points as a program would call them: a
renderer's frame (update list, radiance pass, the consumers' gather), relighting after edits,
animated models put into the world, explicit passes over lists that the host made, batches of
worlds, the relight server, and the gather alone.  Worlds are the seeded terrain worlds of
lum_gb300.worldgen at the sizes of the benchmark and the tests, plus odd ones; volumes start from
a seeded previous state, as in a running program.

  listed()             the cases
  draw(rng)            one more case of the same ranges
  prepare(case, seed)  what a program holds before the call (worlds resident, lists, points)
  run(state)           one pass
  work(case)           bytes and operations a pass cannot do without
  exact(case, seed)    what run returns, in plain torch: the rays are traced in FP32 (the method
                       defines them so: a hit's voxel follows from the FP32 stepping), everything
                       summed, weighted and blended in FP64
"""
from __future__ import annotations

import math

import numpy as np
import torch

import lum_gb300
from lum_gb300 import worldgen

BLEND = 0.1
TYPES = 32
MODEL_SIDE = 32


# ------------------------------------------------------------------------------------- the cases
def listed():
    return [
        # a frame of a thumbnail-sized world: every probe, 64 rays, few consumer points; latency
        _frame("frame_8x8x8", (8, 8, 8), "fp32", (64, 36)),
        # the demo-sized world's frame at a 1280x720 consumer
        _frame("frame_64x64x16", (64, 64, 16), "fp32", (1280, 720), extra=2000),
        # a frame in the reference's own 10-bit volume format while the camera moves: the volume
        # is scrolled by one block first; sizes that are no powers of two
        _frame("frame_scroll_45x38x11", (45, 38, 11), "rgb10a2", (640, 360), scroll=True),
        # a player digs and builds: 0.5% of the blocks change, the probes around them are relit
        {"name": "edits_64x64x16", "kind": "edits", "x": 64, "y": 64, "z": 16, "extra": 2000, "precision": "fp32",
         "rays": 64, "dist": 128.0, "fraction": 0.005, "width": 640, "height": 360},
        # a frame with eight rotated 32^3 voxel models moving through the demo-sized world
        {"name": "models_64x64x16", "kind": "models", "x": 64, "y": 64, "z": 16, "extra": 2000, "precision": "fp32",
         "rays": 64, "dist": 128.0, "meshes": 8, "width": 640, "height": 360},
        # one explicit pass over a host list of 10% of the probes, the volume read back
        _passes("pass_64x64x16_r256", (64, 64, 16), "fp32", 256, 256.0, 1, 0.1, extra=2000),
        # the benchmark's step: 8 passes of 10% of the probes in one call, the volume read back
        _passes("passes8_64x64x16_r256", (64, 64, 16), "fp32", 256, 256.0, 8, 0.1, extra=2000),
        # the largest: every probe of the precision workload's world, FP16 volume
        _passes("pass_all_64x64x32_fp16", (64, 64, 32), "fp16", 256, 256.0, 1, 1.0),
        # odd sizes, a ray count whose subgroups do not divide 8, BF16, a third of the list (time slicing)
        _passes("pass_sliced_45x31x9_r96", (45, 31, 9), "bf16", 96, 128.0, 1, 1.0, size=3, shift=1),
        # many independent worlds of mixed sizes, lists and ray counts per launch
        {"name": "batch_64_worlds", "kind": "batch", "layout": 1, "worlds": 64, "x": 32, "y": 32, "z": 16,
         "precision": "fp32", "dist": 128.0, "runs": 2},
        # relight requests of many worlds, all due at once, served to the end
        {"name": "serve_32_worlds", "kind": "serve", "layout": 1, "worlds": 32, "requests": 128, "blocks": 32768,
         "precision": "fp32", "rays": 64, "dist": 128.0, "radius": 2},
        # the consumers' read of the volume alone, a 1920x1080 view
        {"name": "gather_1920x1080", "kind": "gather", "x": 64, "y": 64, "z": 32, "extra": 0, "precision": "fp32",
         "width": 1920, "height": 1080},
    ]


def _frame(name, dims, precision, view, extra=0, scroll=False, rays=64, dist=128.0):
    return {"name": name, "kind": "frame", "x": dims[0], "y": dims[1], "z": dims[2], "extra": extra,
            "precision": precision, "rays": rays, "dist": dist, "scroll": scroll, "width": view[0], "height": view[1]}


def _passes(name, dims, precision, rays, dist, passes, fraction, extra=0, size=1, shift=0):
    return {"name": name, "kind": "passes", "x": dims[0], "y": dims[1], "z": dims[2], "extra": extra,
            "precision": precision, "rays": rays, "dist": dist, "passes": passes, "fraction": fraction, "size": size,
            "shift": shift}


def draw(rng):
    """One more case: sizes over the listed range (by logarithm), odd ones among them."""
    def side(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def view():
        w = side(48, 1920)
        return w, max(1, w * 9 // 16 + rng.randint(0, 3))

    dims = (side(6, 64), side(6, 64), side(5, 32))
    blocks = dims[0] * dims[1] * dims[2]
    precision = rng.choice(["fp32", "fp32", "fp16", "bf16", "rgb10a2"])
    kind = rng.choice(["frame", "frame", "edits", "models", "passes", "passes", "passes", "batch", "serve", "gather"])
    if kind == "frame":
        c = _frame("", dims, precision, view(), extra=rng.randint(0, blocks // 20), scroll=rng.random() < 0.4,
                   rays=rng.choice([32, 64, 64, 128]), dist=rng.choice([64.0, 128.0, 256.0]))
    elif kind == "edits":
        w, h = view()
        c = {"kind": kind, "x": dims[0], "y": dims[1], "z": dims[2], "extra": rng.randint(0, blocks // 20),
             "precision": precision, "rays": rng.choice([64, 128]), "dist": 128.0,
             "fraction": math.exp(rng.uniform(math.log(0.0005), math.log(0.02))), "width": w, "height": h}
    elif kind == "models":
        w, h = view()
        c = {"kind": kind, "x": max(dims[0], 12), "y": max(dims[1], 12), "z": max(dims[2], 8),
             "extra": rng.randint(0, blocks // 20), "precision": precision, "rays": 64, "dist": 128.0,
             "meshes": rng.randint(1, 12), "width": w, "height": h}
    elif kind == "passes":
        rays = rng.choice([32, 64, 96, 128, 256, 256, 512])
        passes = rng.choice([1, 1, 2, 4, 8, 13])
        most = min(1.0, 3.0e7 / (blocks * rays * passes))
        c = _passes("", dims, precision, rays, rng.choice([64.0, 128.0, 256.0]), passes,
                    most * math.exp(rng.uniform(math.log(0.02), 0.0)), extra=rng.randint(0, blocks // 20),
                    size=rng.choice([1, 1, 1, 2, 3]))
        c["shift"] = rng.randint(0, c["size"] - 1)
    elif kind == "batch":
        c = {"kind": kind, "layout": rng.randint(1, 1 << 30), "worlds": side(8, 96), "x": rng.randint(8, 32),
             "y": rng.randint(8, 32), "z": rng.randint(6, 16), "precision": precision, "dist": 128.0, "runs": rng.randint(1, 2)}
    elif kind == "serve":
        c = {"kind": kind, "layout": rng.randint(1, 1 << 30), "worlds": side(4, 32), "requests": side(16, 128),
             "blocks": side(2048, 32768), "precision": precision, "rays": rng.choice([32, 64, 128]), "dist": 128.0, "radius": rng.randint(1, 3)}
    else:
        w, h = view()
        c = {"kind": kind, "x": dims[0], "y": dims[1], "z": dims[2], "extra": rng.randint(0, blocks // 20),
             "precision": precision, "width": w, "height": h}
    c.pop("name", None)
    return c


# --------------------------------------------------------------------------------------- inputs
def _world(case, seed):
    return worldgen.terrain_world((case["x"], case["y"], case["z"]), seed=seed, n_types=TYPES,
                                  extra_blocks=case.get("extra", 0))


def _volume(world, seed):
    """The volume a running program has: probes of all brightnesses below saturation."""
    return (worldgen.uniform(seed, 77, world.n_blocks * 3) * 0.6).astype(np.float32).reshape(world.grid.shape + (3,))


def _view_points(case, seed):
    """(n, 6) surface points and unit normals in raster order, as a G-buffer holds them: a view over
    the terrain's height range, neighbouring pixels on neighbouring points."""
    w, h = case["width"], case["height"]
    size = np.array([case["x"], case["y"], case["z"]], dtype=np.float64) * 16.0
    a = 2.0 * math.pi * worldgen.uniform(seed, 78, 4)
    v, u = np.meshgrid((np.arange(h) + 0.5) / h, (np.arange(w) + 0.5) / w, indexing="ij")
    px, py = u * size[0], v * size[1]
    amp, kx, ky = 0.1 * size[2], 2.0 * math.pi / 64.0, 2.0 * math.pi / 48.0
    pz = 0.45 * size[2] + amp * np.sin(kx * px + a[0]) * np.cos(ky * py + a[1])
    gx = amp * kx * np.cos(kx * px + a[0]) * np.cos(ky * py + a[1])
    gy = -amp * ky * np.sin(kx * px + a[0]) * np.sin(ky * py + a[1])
    n = 1.0 / np.sqrt(gx * gx + gy * gy + 1.0)
    return np.stack([px, py, pz, -gx * n, -gy * n, n], axis=-1).reshape(-1, 6).astype(np.float32)


def _lists(case, seed):
    dims = (case["x"], case["y"], case["z"])
    return [worldgen.probe_subset(dims, case["fraction"], seed=seed, stream=p) for p in range(case["passes"])]


def _edit_sets(world, case, seed):
    """Two sets of edits at the same blocks: new ids, then the blocks as they were."""
    there = worldgen.edit_request(world.dims, case["fraction"], seed=seed, stream=0, n_types=TYPES)
    back = there.copy()
    back[:, 3] = world.grid[there[:, 2], there[:, 1], there[:, 0]]
    return [there, back]


def _meshes(case, seed, frame):
    """Rotation and place of each model in a frame: a turn about a seeded axis, drifting in x."""
    size = np.array([case["x"], case["y"], case["z"]], dtype=np.float64) * 16.0
    u = worldgen.uniform(seed, 79, 8 * case["meshes"]).reshape(-1, 8)
    out = []
    for row in u:
        axis = row[:3] - 0.5
        axis = axis / np.sqrt((axis * axis).sum())
        half = math.pi * row[3] + 0.02 * frame
        q = tuple(float(np.float32(t)) for t in (*(math.sin(half) * axis), math.cos(half)))
        s = 40.0 + row[4:7] * np.maximum(size - 80.0, 0.0)
        out.append((0, q, (float(np.float32(s[0] + (frame % 16))), float(np.float32(s[1])), float(np.float32(s[2])))))
    return out


def _model(seed):
    u = worldgen.uniform(seed, 80, 2 * MODEL_SIDE ** 3).reshape(2, MODEL_SIDE, MODEL_SIDE, MODEL_SIDE)
    return np.where(u[0] < 0.5, 1 + np.floor(u[1] * 255.0), 0.0).astype(np.uint8)


def _batch_inputs(case, seed):
    """[(world, list, rays)]: sizes uniform per axis from 4 to the case's, lists U(1%, 100%) of the
    probes, 32 to 256 rays (sizes and ray counts are the case's own, contents the seed's)."""
    u = worldgen.uniform(case["layout"], 82, 5 * case["worlds"]).reshape(-1, 5)
    out = []
    for i, row in enumerate(u):
        dims = tuple(4 + int(t * (case[a] - 3)) for t, a in zip(row, "xyz"))
        world = worldgen.terrain_world(dims, seed=1000 * seed + i, n_types=TYPES)
        req = worldgen.probe_subset(dims, 0.01 + 0.99 * row[3], seed=1000 * seed + i)
        out.append((world, req, (32, 64, 128, 256)[int(row[4] * 4)]))
    return out


def _serve_inputs(case, seed):
    """Worlds of lognormal block counts between 512 and the case's, and the requests: a world each
    and U(1%, 5%) of its blocks edited."""
    u = worldgen.uniform(case["layout"], 83, 2 * case["worlds"]).reshape(-1, 2)
    g = np.sqrt(-2.0 * np.log(1.0 - u[:, 0])) * np.cos(2.0 * math.pi * u[:, 1])
    lo, hi = math.log(512), math.log(case["blocks"])
    worlds = []
    for i, b in enumerate(np.clip(np.exp(0.5 * (lo + hi) + 0.25 * (hi - lo) * g), 512, case["blocks"])):
        xy = int(np.clip(round((2.0 * b) ** (1.0 / 3.0)), 8, 64))
        dims = (xy, xy, int(np.clip(round(b / (xy * xy)), 8, 32)))
        worlds.append(worldgen.terrain_world(dims, seed=1000 * seed + i, n_types=TYPES))
    u = worldgen.uniform(seed, 81, 2 * case["requests"]).reshape(-1, 2)
    reqs = []
    for k, (a, b) in enumerate(u):
        i = min(int(a * len(worlds)), len(worlds) - 1)
        reqs.append((i, worldgen.edit_request(worlds[i].dims, 0.01 + 0.04 * b, seed=seed, stream=k, n_types=TYPES)))
    return worlds, reqs


class State(dict):
    """What a program holds; its objects are closed in order when it is dropped."""

    def __del__(self):
        for o in self.get("close", ()):
            o.close()


def _resident(world, case, slots=None, precision=None):
    rw = lum_gb300.RadianceWorld(world.dims, max_block_types=slots or world.palette.shape[0],
                                 precision=precision or case["precision"])
    rw.load(world)
    return rw


def _pinned(shape, dtype):
    return torch.empty(shape, dtype=dtype, pin_memory=True)


def prepare(case, seed):
    kind = case["kind"]
    st = State(kind=kind, case=case, frame=0, seed=seed)
    if kind in ("frame", "edits", "models", "gather"):
        world = _world(case, seed)
        slots = 2048 if kind == "models" else None   # room for the models' temporary blocks
        rw = st["rw"] = _resident(world, case, slots)
        st["close"] = [rw]
        rw.set_radiance(_volume(world, seed))
        st["points"] = torch.from_numpy(_view_points(case, seed)).cuda()
        st["rgb"] = torch.empty((st["points"].shape[0], 3), dtype=torch.float32, device="cuda")
        if kind == "frame" and case["scroll"]:
            rw.set_radiance_shift(1, 0, 0)
        if kind == "edits":
            st["edits"] = _edit_sets(world, case, seed)
        if kind == "models":
            rw.load_model(_model(seed))
            st["static"] = world.palette.shape[0]
            st["meshes"] = [_meshes(case, seed, f) for f in range(32)]
    elif kind == "passes":
        world = _world(case, seed)
        rw = st["rw"] = _resident(world, case)
        st["close"] = [rw]
        rw.set_radiance(_volume(world, seed))
        lists = _lists(case, seed)
        st["counts"] = [int(q.shape[0]) for q in lists]
        packed = st["pin"] = _pinned((sum(st["counts"]), 4), torch.int16)
        packed.numpy()[:] = np.concatenate(lists)
        st["requests"] = packed.numpy()
        st["volume"] = _pinned(world.grid.shape + (3,), torch.float32)
    elif kind == "batch":
        worlds = _batch_inputs(case, seed)
        rws = [_resident(w, case) for w, _, _ in worlds]
        batch = st["batch"] = lum_gb300.RadianceBatch(rws)
        st["close"] = [batch, *rws]
        st["rws"] = rws
        for i, (w, req, rays) in enumerate(worlds):
            rws[i].set_radiance(_volume(w, seed + i))
            batch.set_requests(i, req, lum_gb300.pass_params(rays=rays, max_dist=case["dist"], blend=BLEND))
        sizes = [w.n_blocks for w, _, _ in worlds]
        st["volume"] = _pinned((sum(sizes), 3), torch.float32)
        flat, at = st["volume"].numpy(), np.cumsum([0, *sizes])
        st["parts"] = [flat[at[i]:at[i + 1]] for i in range(len(sizes))]
    else:
        worlds, reqs = _serve_inputs(case, seed)
        rws = [_resident(w, case) for w in worlds]
        srv = st["srv"] = lum_gb300.RadianceServer(precision=case["precision"], radius=case["radius"])
        st["close"] = [srv, *rws]
        for i, (w, rw) in enumerate(zip(worlds, rws)):
            rw.set_radiance(_volume(w, seed + i))
            srv.add_world(rw)
        st["requests"] = [(i, e, _params(case, k)) for k, (i, e) in enumerate(reqs)]
    torch.cuda.synchronize()
    return st


# ------------------------------------------------------------------------------------- one pass
def _params(case, time_seed):
    return lum_gb300.pass_params(rays=case["rays"], max_dist=case["dist"], blend=BLEND, time_seed=time_seed,
                                 size=case.get("size", 1), shift=case.get("shift", 0))


def _gather(st):
    st["rw"].gather_device(st["points"].data_ptr(), st["points"].shape[0], st["rgb"].data_ptr())
    return st["rgb"]


def run(state):
    st, case, kind = state, state["case"], state["kind"]
    f = st["frame"]
    st["frame"] += 1
    if kind == "frame":
        st["rw"].update_radiance(_params(case, f))
        return _gather(st)
    if kind == "gather":
        return _gather(st)
    if kind == "edits":
        edits, rw = st["edits"][f & 1], st["rw"]
        for x, y, z, b in edits.tolist():
            rw.set_world_block(x, y, z, b)
        dirty = rw.build_dirty_list(edits, 2)
        rw.radiance_pass(dirty, _params(case, f))
        return _gather(st)
    if kind == "models":
        st["rw"].blockify(st["static"], st["meshes"][f % 32])
        st["rw"].update_radiance(_params(case, f))
        return _gather(st)
    if kind == "passes":
        n = len(st["counts"])
        if n == 1:
            st["rw"].radiance_pass(st["requests"], _params(case, f))
        else:
            st["rw"].radiance_passes_packed(st["requests"], st["counts"], [_params(case, n * f + p) for p in range(n)])
        return st["rw"].get_radiance(st["volume"].numpy())
    if kind == "batch":
        for k in range(case["runs"]):
            st["batch"].run(case["runs"] * f + k)
        st["batch"].synchronize()
        for rw, part in zip(st["rws"], st["parts"]):
            rw.get_radiance(part)
        return st["volume"].numpy()
    srv = st["srv"]
    for i, edits, p in st["requests"]:
        srv.submit(i, edits, p)
    srv.run()
    done = srv.poll()
    probes = done["probes"][np.argsort(done["request"])].astype(np.int32)
    return probes, np.concatenate([srv.get_radiance(i).reshape(-1, 3) for i in range(case["worlds"])])


# ----------------------------------------------------------------------------------------- work
_STRIDE = {"fp32": 16, "fp16": 8, "bf16": 8, "rgb10a2": 4}
# Operations of a ray that no implementation can leave out, for the worlds here: its set-up (two
# hashes, a normalisation, about 90), 15 coarse steps of about 30, and refine, taps and shading
# (about 200); of a gathered point: 8 probes of about 35.
_RAY_FLOPS, _POINT_FLOPS = 90 + 15 * 30 + 200, 8 * 35


def work(case):
    kind = case["kind"]
    stride = _STRIDE[case["precision"]]
    pal = (TYPES + 1) * 4096
    if kind == "batch":
        blocks = case["worlds"] * ((4 + case["x"]) / 2) * ((4 + case["y"]) / 2) * ((4 + case["z"]) / 2)
        rays = 0.5 * blocks * 120.0
        return {"bytes": case["runs"] * (blocks * (2 + 2 * stride + 4) + case["worlds"] * pal) + 12 * blocks,
                "flops": case["runs"] * rays * _RAY_FLOPS}
    if kind == "serve":
        mean = math.sqrt(512.0 * case["blocks"]) * 1.6
        side = 2 * case["radius"] + 1
        probes = mean * min(1.0, 0.03 * side ** 3 * 0.7)
        return {"bytes": case["requests"] * (mean * 0.03 * 8 + probes * (8 + 2 * stride) + mean * 2 + pal) +
                case["worlds"] * mean * 12, "flops": case["requests"] * probes * case["rays"] * _RAY_FLOPS}
    blocks = case["x"] * case["y"] * case["z"]
    points = case.get("width", 0) * case.get("height", 0)
    out = points * (24 + 12) + (12 * blocks if kind == "passes" else 0)
    if kind == "gather":
        return {"bytes": blocks * stride + out, "flops": points * _POINT_FLOPS}
    probes = {"frame": 0.55 * blocks, "models": 0.55 * blocks,
              "edits": blocks * min(1.0, 125 * case.get("fraction", 0) * 0.8),
              "passes": case.get("passes", 1) * case.get("fraction", 0) * blocks / case.get("size", 1)}[kind]
    models = case.get("meshes", 0) * (MODEL_SIDE ** 3 + 27 * 4096)
    return {"bytes": blocks * 2 + pal + models + blocks * stride + probes * (8 + stride) + out,
            "flops": probes * case["rays"] * _RAY_FLOPS + points * _POINT_FLOPS}


# ---------------------------------------------------------------------- the same in plain torch
_CHUNK = 1 << 22   # rays traced at a time


class _Exact:
    """One world: the grid and palette as tensors, the volume in FP64."""

    def __init__(self, grid, palette, materials, volume):
        self.Z, self.Y, self.X = grid.shape
        self.grid = torch.from_numpy(grid.reshape(-1).astype(np.int64)).cuda()
        self.pal = torch.from_numpy(palette.reshape(-1).astype(np.int64)).cuda()
        self.slots = palette.shape[0]
        self.mats = torch.from_numpy(materials.astype(np.float64)).cuda()
        self.vol = torch.from_numpy(volume.astype(np.float64).reshape(-1, 3)).cuda()

    def voxels(self, ip):
        """Block id and voxel value at integer voxel coordinates (n, 3); outside the grid block 0."""
        b = torch.div(ip, 16, rounding_mode="trunc")
        size = torch.tensor([self.X, self.Y, self.Z], device=ip.device)
        inside = ((b >= 0) & (b < size)).all(1) & (ip > -16).all(1)
        at = torch.where(inside, b[:, 0] + self.X * (b[:, 1] + self.Y * b[:, 2]), 0)
        block = torch.where(inside, self.grid[at], 0)
        slot = torch.where(block < 0, block + 64, block)
        has = (block >= -63) & (slot < self.slots)
        v = ip & 15
        value = torch.where(has, self.pal[torch.where(has, slot, 0) * 4096 + v[:, 0] + 16 * v[:, 1] + 256 * v[:, 2]], 0)
        return block, value

    def sample(self, u):
        """Trilinear, repeating, at u in [0, 1) of the volume's size."""
        size = torch.tensor([self.X, self.Y, self.Z], device=u.device)
        t = u.double() * size - 0.5
        lo = torch.floor(t)
        w = t - lo
        lo = lo.long()
        total = torch.zeros((u.shape[0], 3), dtype=torch.float64, device=u.device)
        for corner in range(8):
            o = torch.tensor([corner & 1, corner >> 1 & 1, corner >> 2], device=u.device)
            q = torch.remainder(lo + o, size)
            k = torch.where(o.bool(), w, 1.0 - w).prod(1)
            total += k[:, None] * self.vol[q[:, 0] + self.X * (q[:, 1] + self.Y * q[:, 2])]
        return total

    def relight(self, req, rays, dist, seed, size=1, shift=0):
        """One pass over the list: the listed probes blended with their rays' mean light."""
        groups = req.shape[0] // size
        q = torch.from_numpy(np.ascontiguousarray(req[shift::size][:groups, :3]).astype(np.int64)).cuda()
        light = torch.empty((groups, 3), dtype=torch.float64, device="cuda")
        step = max(1, _CHUNK // rays)
        for g in range(0, groups, step):
            light[g:g + step] = self.light(q[g:g + step], g, rays, dist, seed)
        at = q[:, 0] + self.X * (q[:, 1] + self.Y * q[:, 2])
        new = self.vol.clone()
        new[at] = (self.vol[at].clamp(0.0, 1.0) * (1.0 - BLEND) + light * BLEND).clamp(0.0, 1.0)
        self.vol = new

    def light(self, q, first, rays, dist, seed):
        n = q.shape[0]
        o, d = _rays(q, first, rays, seed)
        size = torch.tensor([self.X, self.Y, self.Z], device="cuda")
        far = (size * 16).float()
        inv = 1.0 / d
        hit_f = torch.full((n * rays,), -1.0, dtype=torch.float32, device="cuda")
        live = torch.arange(n * rays, device="cuda")
        f = torch.zeros(n * rays, dtype=torch.float32, device="cuda")
        oo, dd, ii = o, d, inv
        for _ in range(int(2.0 * dist) + 2):
            f = f + 0.5
            p = oo + dd * f[:, None]
            block, value = self.voxels(p.trunc().long())
            corner = torch.trunc(p * 0.0625) * 16.0 + torch.where(dd > 0, 16.0, 0.0)
            t = corner * ii + (-p) * ii
            skip = torch.maximum(t.amin(1), torch.full_like(f, 0.01))
            f = torch.where(block == 0, f + skip, f)
            solid = value != 0
            hit_f[live[solid]] = f[solid]
            on = ~(solid | (p < 0).any(1) | (p >= far).any(1) | (f >= dist))
            live, f, oo, dd, ii = live[on], f[on], oo[on], dd[on], ii[on]
            if live.numel() == 0:
                break
        out = torch.zeros((n * rays, 3), dtype=torch.float64, device="cuda")
        gl = torch.tensor([0.5, 0.5, -0.9], dtype=torch.float64, device="cuda")
        gl = gl / gl.pow(2).sum().sqrt()
        g = -(d.double() @ gl)
        sun = torch.tensor([0.9, 0.9, 0.6], dtype=torch.float64, device="cuda") * 3.0
        sky = torch.tensor([0.53, 0.81, 0.92], dtype=torch.float64, device="cuda") * 0.1
        out = torch.where((g > 0.95)[:, None], g[:, None] * sun, 0.0) + sky
        hits = torch.nonzero(hit_f >= 0).reshape(-1)
        out[hits] = self.shade(o[hits], d[hits], inv[hits], hit_f[hits])
        return out.reshape(n, rays, 3).mean(1)

    def shade(self, o, d, inv, f):
        """The refine stepping to the voxel's face (at most 5 steps), its material, the volume there."""
        p = o + d * (f - 1.5)[:, None]
        way = torch.where(d > 0, 1, -1)
        c = (torch.floor(p) - p) / d
        tm, td = torch.maximum(c, c + inv), inv.abs()
        v = p.trunc().long()
        fs = torch.zeros_like(p)
        value = self.voxels(v)[1]
        for _ in range(5):
            go = value == 0
            axis = torch.stack([(tm[:, 0] <= tm[:, 1]) & (tm[:, 0] <= tm[:, 2]),
                                (tm[:, 0] >= tm[:, 1]) & (tm[:, 1] <= tm[:, 2]),
                                (tm[:, 2] <= tm[:, 0]) & (tm[:, 2] <= tm[:, 1])], dim=1) & go[:, None]
            fs = torch.where(go[:, None], axis.float(), fs)
            v = v + torch.where(axis, way, 0)
            tm = torch.where(axis, tm + td, tm)
            value = torch.where(go, self.voxels(v)[1], value)
        t = (tm - td) * fs
        fr = (t[:, 0] + t[:, 1]) + t[:, 2]
        place = ((o + fr[:, None] * d) + (-(way * fs)) * 16.0) * 0.0625
        size = torch.tensor([self.X, self.Y, self.Z], device="cuda").float()
        m = self.mats[value]
        return self.sample((place + 0.5) / size) * m[:, :3] + m[:, :3] * m[:, 4:5]

    def gather(self, points):
        """The consumers' read: the 8 probes around a point, weighted by distance and direction."""
        out = []
        for pts in torch.from_numpy(points).cuda().split(1 << 20):
            x, nrm = pts[:, :3].double(), pts[:, 3:].double()
            size = torch.tensor([self.X, self.Y, self.Z], device="cuda")
            z = torch.div(torch.floor(pts[:, :3] - 8.0).long(), 16, rounding_mode="trunc").clamp(min=0)
            z = torch.minimum(z, size)
            c = z.double() * 16.0 + 8.0
            a = ((x - c) / 16.0).clamp(0.0, 1.0)
            tw = torch.zeros(pts.shape[0], dtype=torch.float64, device="cuda")
            tot = torch.zeros((pts.shape[0], 3), dtype=torch.float64, device="cuda")
            for corner in range(8):
                off = torch.tensor([corner & 1, corner >> 1 & 1, corner >> 2], device="cuda")
                to = c + off * 16.0 - x
                to = to / to.pow(2).sum(1, keepdim=True).sqrt()
                w = torch.where(off.bool(), a, 1.0 - a).prod(1) * (to * nrm).sum(1).clamp(0.1, 1.0)
                w = w.clamp(min=1e-7)
                q = torch.minimum(z + off, size)
                inside = (q < size).all(1)
                at = torch.where(inside, q[:, 0] + self.X * (q[:, 1] + self.Y * q[:, 2]), 0)
                tot += w[:, None] * torch.where(inside[:, None], self.vol[at].clamp(0.0, 2.0), 0.0)
                tw += w
            out.append(tot / tw[:, None])
        return torch.cat(out)


def _hash3(x, y, z):
    k, m = 1103515245, 0xFFFFFFFF
    for _ in range(3):
        x, y, z = ((x >> 8) ^ y) * k & m, ((y >> 8) ^ z) * k & m, ((z >> 8) ^ x) * k & m
    return torch.stack([x, y, z], dim=1).float() * 2.0 ** -32


def _directions(rays):
    f = np.float32
    i = np.arange(rays, dtype=np.float32)
    golden = np.sqrt(f(5.0)) * f(0.5) + f(0.5)
    a = i * (golden - f(1.0))
    phi = f(2.0) * f(math.pi) * (a - np.floor(a))
    cos_t = f(1.0) - (f(2.0) * i + f(1.0)) * (f(1.0) / f(rays))
    sin_t = np.sqrt(np.clip(f(1.0) - cos_t * cos_t, f(0.0), f(1.0)))
    c, s = np.cos(phi.astype(np.float64)).astype(f), np.sin(phi.astype(np.float64)).astype(f)
    return np.stack([c * sin_t, s * sin_t, cos_t], axis=1)


def _rays(q, first, rays, seed):
    """Origins and directions of every ray of probes q (their list positions start at `first`)."""
    n = q.shape[0]
    r = torch.arange(rays, device="cuda").repeat(n)
    g = torch.arange(first, first + n, device="cuda").repeat_interleave(rays)
    s = torch.full_like(r, seed & 0xFFFFFFFF)
    sx = (g * rays + r + seed) & 0xFFFFFFFF
    base = torch.from_numpy(_directions(rays)).cuda()[r]
    j = base + (_hash3(sx, s, s) - 0.5) * 0.2
    length = torch.sqrt((j[:, 0] * j[:, 0] + j[:, 1] * j[:, 1]) + j[:, 2] * j[:, 2])
    d = j * (1.0 / length)[:, None]
    o = (q.float() * 16.0 + 8.0).repeat_interleave(rays, 0) + d * 6.0
    o = o + (_hash3((sx + 1) & 0xFFFFFFFF, s, s) - 0.5) * 2.0
    return o, torch.where((r & 1).bool()[:, None], -d, d)


def _update_list(grid):
    """Blocks whose 3x3x3 neighbourhood (clamped at the border) has a positive sum of ids."""
    g = np.pad(grid.astype(np.int64), 1, mode="edge")
    Z, Y, X = grid.shape
    total = sum(g[a:a + Z, b:b + Y, c:c + X] for a in range(3) for b in range(3) for c in range(3))
    z, y, x = np.nonzero(total > 0)
    return np.stack([x, y, z, np.zeros_like(x)], axis=1)


def _dirty(dims, edits, radius):
    X, Y, Z = dims
    mask = np.zeros((Z, Y, X), dtype=bool)
    for x, y, z in edits[:, :3].tolist():
        mask[max(z - radius, 0):z + radius + 1, max(y - radius, 0):y + radius + 1,
             max(x - radius, 0):x + radius + 1] = True
    z, y, x = np.nonzero(mask)
    return np.stack([x, y, z, np.zeros_like(x)], axis=1)


def _edited(grid, edits):
    g = grid.copy()
    for x, y, z, b in edits.tolist():
        g[z, y, x] = b
    return g


def _with_models(world, meshes, model, slots):
    """The frame's grid and palette: blocks under a model's box get temporary slots that hold the
    block and the model's voxels over it (FP32 transforms, models and voxels in order)."""
    grid = world.grid.astype(np.int64).copy()
    Z, Y, X = grid.shape
    static = world.palette.shape[0]
    pal = np.zeros((slots, 16, 16, 16), dtype=np.uint8)
    pal[:static] = world.palette
    f, count, boxes = np.float32, static, []
    for _, q, s in meshes:
        x, y, z, w = (f(v) for v in q)
        m = np.array([[1 - 2 * (y * y + z * z), 2 * (x * y + w * z), 2 * (x * z - w * y)],
                      [2 * (x * y - w * z), 1 - 2 * (x * x + z * z), 2 * (y * z + w * x)],
                      [2 * (x * z + w * y), 2 * (y * z - w * x), 1 - 2 * (x * x + y * y)]], dtype=f)   # m[col][row]
        corners = np.array([[a, b, c] for a in (0, 1) for b in (0, 1) for c in (0, 1)], dtype=np.float64)
        at = (corners * (MODEL_SIDE - 1) @ m.astype(np.float64) + np.array(s, dtype=np.float64)).astype(f)
        lo, hi = at.min(0), at.max(0)
        boxes.append((m, np.array(s, dtype=np.float64), lo, hi))
        size = np.array([X, Y, Z])
        b0 = np.clip(np.trunc((np.trunc(lo) - 1) / 16), 0, size - 1).astype(int)
        b1 = np.clip(np.trunc((np.trunc(hi) + 1) / 16), 0, size - 1).astype(int)
        for bz in range(b0[2], b1[2] + 1):
            for by in range(b0[1], b1[1] + 1):
                for bx in range(b0[0], b1[0] + 1):
                    if grid[bz, by, bx] < static:
                        pal[count] = pal[grid[bz, by, bx]]
                        grid[bz, by, bx] = count
                        count += 1
    for m, s, lo, hi in boxes:
        first = np.floor(lo).astype(int)
        n = (np.ceil(hi).astype(int) - first + 3) // 4 * 4
        gz, gy, gx = np.meshgrid(np.arange(n[2]), np.arange(n[1]), np.arange(n[0]), indexing="ij")
        p = np.stack([gx, gy, gz], axis=-1).reshape(-1, 3)
        p = (p.astype(f) + f(0.5)) + first.astype(f)
        back = (-(m.astype(np.float64) @ s)).astype(f)
        v = np.stack([((m[k, 0] * p[:, 0] + m[k, 1] * p[:, 1]) + m[k, 2] * p[:, 2]) + back[k] for k in range(3)],
                     axis=1)
        v, ip = np.trunc(v).astype(int), np.trunc(p).astype(int)
        b = np.trunc(ip / 16).astype(int)
        ok = ((b >= 0) & (b < [X, Y, Z])).all(1) & ((v >= 0) & (v < MODEL_SIDE)).all(1)
        ip, b, v = ip[ok], b[ok], v[ok]
        slot = grid[b[:, 2], b[:, 1], b[:, 0]]
        value = model[v[:, 2], v[:, 1], v[:, 0]]
        ok = (slot >= static) & (value != 0)
        k = ip[ok] & 15
        pal[slot[ok], k[:, 2], k[:, 1], k[:, 0]] = value[ok]   # in order: the last one stays
    return grid, pal


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        out = []
        for i, (w, req, rays) in enumerate(_batch_inputs(case, seed)):
            e = _Exact(w.grid, w.palette, w.materials, _volume(w, seed + i))
            for k in range(case["runs"]):
                e.relight(req, rays, case["dist"], k)
            out.append(e.vol)
        return torch.cat(out)
    if kind == "serve":
        worlds, reqs = _serve_inputs(case, seed)
        grids = [w.grid for w in worlds]
        es = [_Exact(w.grid, w.palette, w.materials, _volume(w, seed + i)) for i, w in enumerate(worlds)]
        for k, (i, edits) in enumerate(reqs):
            grids[i] = _edited(grids[i], edits)
            es[i].grid = torch.from_numpy(grids[i].reshape(-1).astype(np.int64)).cuda()
            es[i].relight(_dirty(worlds[i].dims, edits, case["radius"]), case["rays"], case["dist"], k)
        return None, torch.cat([e.vol for e in es])
    world = _world(case, seed)
    grid, pal = world.grid, world.palette
    if kind == "edits":
        edits = _edit_sets(world, case, seed)[0]
        grid = _edited(grid, edits)
    if kind == "models":
        grid, pal = _with_models(world, _meshes(case, seed, 0), _model(seed), 2048)
    e = _Exact(grid, pal, world.materials, _volume(world, seed))
    if kind == "passes":
        for p, req in enumerate(_lists(case, seed)):
            e.relight(req, case["rays"], case["dist"], p, case["size"], case["shift"])
        return e.vol.reshape(world.grid.shape + (3,))
    if kind == "frame" and case["scroll"]:
        v = e.vol.reshape(world.grid.shape + (3,))
        e.vol = torch.cat([v[:, :, 1:], v[:, :, -1:]], dim=2).reshape(-1, 3)
    if kind in ("frame", "models"):
        e.relight(_update_list(grid), case["rays"], case["dist"], 0)
    if kind == "edits":
        e.relight(_dirty(world.dims, edits, 2), case["rays"], case["dist"], 0)
    return e.gather(_view_points(case, seed))
