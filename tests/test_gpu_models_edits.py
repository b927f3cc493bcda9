"""Block edits while a frame of models is in the world: the frame gives way to the changed world (whose next pass
equals the same world loaded whole), the next models' call puts its models into it; with block ids below and
inside the models' range of palette slots, and frames of different ranges."""
import numpy as np
import pytest

from lum_gb300 import worldgen
from tests.helpers import random_prev
from tests.test_gpu_world_edits import _params, _same

pytestmark = pytest.mark.gpu

DIMS = (13, 11, 6)
SLOTS = 400


def _meshes(k, n):
    rng = np.random.default_rng(k)
    out = []
    for _ in range(n):
        q = rng.normal(size=4)
        s = rng.random(3) * np.array(DIMS) * 13.0
        out.append((0, tuple(float(np.float32(t)) for t in q / np.linalg.norm(q)), tuple(float(np.float32(t)) for t in s)))
    return out


# what an edit brings in, relative to the lowest id the models take: an id of the world, air, one without a slot; an id of
# the models' range, a negative id whose slot is in it
@pytest.mark.parametrize("ids", [(-3, -7), (-2, 0, 9000), (2, -2), ("negative", -1)])
@pytest.mark.parametrize("end", ["frame", "batch", "server"])
def test_edits_beside_models(ids, end):
    import lum_gb300
    import oracle
    w = worldgen.terrain_world(DIMS, seed=76, n_types=20)
    static = w.palette.shape[0]
    model = ((np.random.default_rng(1).random((24, 30, 20)) < 0.6) * 5).astype(np.uint8)
    new = [{"negative": static + 3 - 64, 0: 0, 9000: 9000}.get(i, static + i if not isinstance(i, str) else 0) for i in ids]
    with lum_gb300.RadianceWorld(DIMS, max_block_types=SLOTS) as rw:
        rw.load(w)
        rw.load_model(model)
        prev = random_prev(w)
        rw.set_radiance(prev)
        grid = w.grid.copy()
        rng = np.random.default_rng(7)

        def edit(n):
            for _ in range(n):
                x, y, z = (int(rng.integers(d)) for d in DIMS)
                b = int(rng.choice(new))
                rw.set_world_block(x, y, z, b)
                grid[z, y, x] = b

        def models(k, n, first):
            nonlocal prev
            pal = np.zeros((SLOTS, 16, 16, 16), np.uint8)
            pal[:static] = w.palette
            meshes = _meshes(k, n)
            ref_grid, ref_pal = oracle.blockify(grid, pal, first, [model], meshes)
            rw.blockify(first, meshes)
            assert np.array_equal(rw.get_world(), ref_grid)
            # (slots below `first` keep what a frame of a lower range left there)
            assert np.array_equal(rw.get_block_palette()[first:], ref_pal[first:])
            rw.update_radiance(_params(k))
            if first == static:
                fw = worldgen.World(grid=ref_grid, palette=ref_pal, materials=w.materials)
                prev, _, _ = oracle.radiance_pass(fw, oracle.update_list(fw), prev=prev, rays=32, max_dist=96.0, blend=0.3, time_seed=k)
                assert rw.get_radiance().tobytes() == prev.tobytes()

        models(0, 4, static)
        edit(9)
        prev = _same(rw, grid, w, prev, 1, True)      # the frame is gone, the edits are there
        models(2, 3, static)
        edit(3)
        models(3, 5, static)                          # an edit and the next frame before a pass
        edit(1)
        edit(0)
        prev = _same(rw, grid, w, prev, 4, False)
        edit(2)                                       # no frame in between
        prev = _same(rw, grid, w, prev, 5, True)
        models(6, 4, static + 6)                      # a range that starts higher, after a lower one
        edit(4)
        rw.set_radiance(prev)
        prev = _same(rw, grid, w, prev, 7, True)
        models(8, 2, static)
        edit(5)
        if end == "frame":
            prev = _same(rw, grid, w, prev, 9, True)
            rw.set_world_block(4, 4, 2, static + 1)   # an id that the frames before had used for models
            grid[2, 4, 4] = static + 1
            _same(rw, grid, w, prev, 10, True)
            return
        req = worldgen.all_probes(DIMS)
        pal = np.zeros((SLOTS, 16, 16, 16), np.uint8)
        pal[:static] = w.palette
        fw = worldgen.World(grid=grid, palette=pal, materials=w.materials)
        p = dict(rays=32, max_dist=96.0, blend=0.3)
        if end == "batch":
            ref, _, _ = oracle.radiance_pass(fw, req, prev=prev, time_seed=9, **p)
            with lum_gb300.RadianceBatch([rw]) as b:
                b.set_requests(0, req, lum_gb300.pass_params(**p))
                b.run(9)
                b.synchronize()
                assert rw.get_radiance().tobytes() == ref.tobytes()
            return
        prev = _same(rw, grid, w, prev, 9, True)      # no frame, no edits left: the server starts from here
        late = [(x, 3, 4, b) for x, b in zip(range(12), [static + 1, static + 30, 5, static - 1] * 3)]
        for x, y, z, b in late:
            grid[z, y, x] = b
        with lum_gb300.RadianceServer(radius=15) as s:
            s.add_world(rw)
            s.submit(0, np.array(late, np.int16), lum_gb300.pass_params(time_seed=11, **p))
            s.run()
            dirty = lum_gb300.dirty_probes(DIMS, np.array(late, np.int16), 15)
            ref, _, _ = oracle.radiance_pass(fw, dirty, prev=prev, time_seed=11, **p)
            assert s.get_radiance(0).tobytes() == ref.tobytes()
