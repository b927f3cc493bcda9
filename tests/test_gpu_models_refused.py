"""A refused models' call leaves the context as it was: without a frame of models in the world, block edits
after it show at once and reach the next pass; with one, the frame stays."""
import numpy as np
import pytest

from lum_gb300 import worldgen
from tests.helpers import random_prev
from tests.test_gpu_world_edits import _same

pytestmark = pytest.mark.gpu

UPRIGHT = (0.0, 0.0, 0.0, 1.0)


# too few block types for the model's blocks; a mesh of 2^32 world voxels or more (by a quaternion that
# is not of unit length)
@pytest.mark.parametrize("dims,slots,refused", [((13, 11, 6), 3, (0, UPRIGHT, (16.0, 32.0, 40.0))),
                                                ((3, 3, 2), 18, (1, (100.0, 100.0, 100.0, 100.0), (20.0, 20.0, 20.0)))])
@pytest.mark.parametrize("models_before", [False, True])
def test_refused_models(dims, slots, refused, models_before):
    import lum_gb300
    w = worldgen.terrain_world(dims, seed=75, n_types=20)
    static = w.palette.shape[0]
    with lum_gb300.RadianceWorld(dims, max_block_types=static + slots) as rw:
        rw.load(w)
        prev = random_prev(w)
        rw.set_radiance(prev)
        rw.load_model(np.full((40, 40, 40), 9, np.uint8))
        rw.load_model(np.full((2, 2, 2), 9, np.uint8))
        if models_before:
            rw.blockify(static, [(1, UPRIGHT, (20.0, 20.0, 20.0))])
            frame = rw.get_world()
            assert not np.array_equal(frame, w.grid)
        with pytest.raises(lum_gb300.LumRadError):
            rw.blockify(static, [refused])
        if models_before:
            assert np.array_equal(rw.get_world(), frame)
            return
        grid = w.grid.copy()
        assert np.array_equal(rw.get_world(), grid)
        for x, y, z in ((1, 2, dims[2] - 1), (dims[0] - 1, 0, 0)):
            grid[z, y, x] = 9 if grid[z, y, x] != 9 else 8
            rw.set_world_block(x, y, z, int(grid[z, y, x]))
        assert np.array_equal(rw.get_world(), grid)
        _same(rw, grid, w, prev, 0, True)
