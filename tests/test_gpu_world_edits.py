"""Worlds changed block by block between passes (set_world_block), new block ids among them, and models
put into the world frame after frame: each pass against the same world loaded whole."""
import numpy as np
import pytest

from lum_gb300 import worldgen
from tests.helpers import random_prev

pytestmark = pytest.mark.gpu


def _params(k):
    import lum_gb300
    return lum_gb300.pass_params(rays=32, max_dist=96.0, blend=0.3, time_seed=k)


def _same(rw, grid, w, prev, k, frame):
    """One pass (a frame's or an explicit one) on rw and on a fresh context of that grid; the volume."""
    import lum_gb300
    req = worldgen.all_probes(w.dims)
    with lum_gb300.RadianceWorld(w.dims, max_block_types=rw.max_block_types) as b:
        for slot in range(w.palette.shape[0]):
            b.load_block(slot, w.block_voxels(slot))
        b.upload_block_palette()
        b.load_materials(w.materials)
        b.upload_material_palette()
        b.load_world(grid)
        b.set_radiance(prev)
        for x in (rw, b):
            x.update_radiance(_params(k)) if frame else x.radiance_pass(req, _params(k))
        got, ref = rw.get_radiance(), b.get_radiance()
        assert np.array_equal(rw.get_world(), grid)
        assert got.tobytes() == ref.tobytes()
        assert rw.pass_stats()["steps"] == b.pass_stats()["steps"]
    return got


@pytest.mark.parametrize("types", [40, 300])   # one and two bytes per compact id
@pytest.mark.parametrize("frame", [False, True])
def test_edits_between_passes(types, frame):
    import lum_gb300
    dims = (14, 9, 7)
    w = worldgen.terrain_world(dims, seed=71, n_types=types)
    w.grid = np.minimum(w.grid, 5).astype(np.int16)     # most ids appear only with the edits
    rng = np.random.default_rng(types)
    with lum_gb300.RadianceWorld(dims, max_block_types=w.palette.shape[0]) as rw:
        rw.load(w)
        prev = random_prev(w)
        rw.set_radiance(prev)
        grid = w.grid.copy()
        for k, n in enumerate((1, 7, 0, 60, 400, 3)):    # 400: more than an eighth of the world
            for _ in range(n):
                x, y, z = (int(rng.integers(d)) for d in dims)
                b = int(rng.integers(-70, types + 3))
                rw.set_world_block(x, y, z, b)
                rw.set_world_block(x, y, z, b)
                grid[z, y, x] = b
                assert rw.get_world_block(x, y, z) == b
            prev = _same(rw, grid, w, prev, k, frame)


def test_edits_before_a_new_palette():
    import lum_gb300
    dims = (11, 8, 6)
    w = worldgen.terrain_world(dims, seed=73, n_types=20)
    grid = w.grid.copy()
    with lum_gb300.RadianceWorld(dims, max_block_types=w.palette.shape[0]) as rw:
        rw.load(w)
        prev = random_prev(w)
        rw.set_radiance(prev)
        prev = _same(rw, grid, w, prev, 0, True)
        for x, y, z, b in ((3, 3, 5, 9), (9, 1, 4, 4), (0, 7, 0, 0)):   # the first two above the terrain
            rw.set_world_block(x, y, z, b)
            grid[z, y, x] = b
        rw.upload_block_palette()
        _same(rw, grid, w, prev, 1, True)


def test_edits_then_batch_and_server():
    import lum_gb300
    import oracle
    w = worldgen.small_world()
    req = worldgen.all_probes(w.dims)
    prev = random_prev(w)
    grid = w.grid.copy()
    grid[2, 3, 4], grid[5, 1, 1] = 9, 0
    edited = worldgen.World(grid=grid, palette=w.palette, materials=w.materials)
    p = dict(rays=32, max_dist=96.0, blend=0.3)
    ref, _, _ = oracle.radiance_pass(edited, req, prev=prev, time_seed=4, **p)
    for kind in ("batch", "server"):
        with lum_gb300.RadianceWorld(w.dims, max_block_types=w.palette.shape[0]) as rw:
            rw.load(w)
            rw.set_radiance(prev)
            rw.radiance_pass(req[:1], lum_gb300.pass_params(time_seed=9, **dict(p, blend=0.0)))
            rw.set_world_block(4, 3, 2, 9)
            rw.set_world_block(1, 1, 5, 0)
            if kind == "batch":
                with lum_gb300.RadianceBatch([rw]) as b:
                    b.set_requests(0, req, lum_gb300.pass_params(**p))
                    b.run(4)
                    b.synchronize()
                    assert rw.get_radiance().tobytes() == ref.tobytes()
            else:
                with lum_gb300.RadianceServer(radius=15) as s:
                    s.add_world(rw)
                    s.submit(0, np.array([[4, 3, 2, 9]], np.int16), lum_gb300.pass_params(time_seed=4, **p))
                    s.run()
                    assert s.get_radiance(0).tobytes() == ref.tobytes()


@pytest.mark.parametrize("n_slots", [120, 700])   # the second run needs two bytes per compact id
def test_models_frame_after_frame(n_slots):
    import lum_gb300
    import oracle
    dims = (13, 11, 6)
    w = worldgen.terrain_world(dims, seed=72, n_types=20)
    static = w.palette.shape[0]
    rng = np.random.default_rng(5)
    models = [((rng.random((9, 12, 20)) < 0.6) * rng.integers(1, 256, (9, 12, 20))).astype(np.uint8),
              ((rng.random((30, 24, 28)) < 0.5) * rng.integers(1, 256, (30, 24, 28))).astype(np.uint8)]
    with lum_gb300.RadianceWorld(dims, max_block_types=n_slots) as rw:
        rw.load(w)
        for m in models:
            rw.load_model(m)
        prev = random_prev(w)
        rw.set_radiance(prev)
        grid = w.grid.copy()
        for k in range(7):
            meshes = []
            for i in range((3, 0, 26, 1, 5, 2, 2)[k]):   # 26: two launches of the map
                q = rng.normal(size=4)
                q = tuple(float(np.float32(t)) for t in q / np.linalg.norm(q))
                far = n_slots > 256 or k != 2
                s = rng.random(3) * np.array(dims) * (14.0 if far else 2.0)
                meshes.append((int(i % 2), q, tuple(float(np.float32(t)) for t in s)))
            if k == 4:                                   # the origin world changes between frames
                rw.set_world_block(2, 2, 2, 7)
                grid[2, 2, 2] = 7
            pal = np.zeros((n_slots, 16, 16, 16), np.uint8)
            pal[:static] = w.palette
            ref = oracle.blockify(grid, pal, static, models, meshes)
            if ref is None:                              # more blocks than slots: refused, the world stays
                before = grid if k == 4 else rw.get_world()   # (but a changed origin world replaces the frame)
                with pytest.raises(lum_gb300.LumRadError):
                    rw.blockify(static, meshes)
                assert np.array_equal(rw.get_world(), before)
                continue
            ref_grid, ref_pal = ref
            rw.blockify(static, meshes)
            assert np.array_equal(rw.get_world(), ref_grid)
            assert np.array_equal(rw.get_block_palette(), ref_pal)
            fw = worldgen.World(grid=ref_grid, palette=ref_pal, materials=w.materials)
            rw.update_radiance(_params(k))
            prev, _, _ = oracle.radiance_pass(fw, oracle.update_list(fw), prev=prev, rays=32, max_dist=96.0, blend=0.3, time_seed=k)
            assert rw.get_radiance().tobytes() == prev.tobytes()


def test_models_then_batch():
    """A batch runs on its own stream, right after the models' call returned."""
    import lum_gb300
    import oracle
    w = worldgen.terrain_world((13, 11, 6), seed=74, n_types=20)
    static, n_slots = w.palette.shape[0], 700
    model = np.full((30, 24, 28), 77, np.uint8)
    req = worldgen.all_probes(w.dims)
    p = dict(rays=32, max_dist=96.0, blend=0.3)
    with lum_gb300.RadianceWorld(w.dims, max_block_types=n_slots) as rw:
        rw.load(w)
        rw.load_model(model)
        prev = random_prev(w)
        rw.set_radiance(prev)
        with lum_gb300.RadianceBatch([rw]) as b:
            for k in range(3):
                meshes = [(0, (1.0, 0.0, 0.0, 0.0), (16.0 * i + 3.0 * k, 40.0, 30.0)) for i in range(8)]
                b.set_requests(0, req, lum_gb300.pass_params(**p))
                rw.blockify(static, meshes)
                b.run(k)
                pal = np.zeros((n_slots, 16, 16, 16), np.uint8)
                pal[:static] = w.palette
                grid, pal = oracle.blockify(w.grid, pal, static, [model], meshes)
                fw = worldgen.World(grid=grid, palette=pal, materials=w.materials)
                prev, _, _ = oracle.radiance_pass(fw, req, prev=prev, time_seed=k, **p)
                b.synchronize()
                assert rw.get_radiance().tobytes() == prev.tobytes()
