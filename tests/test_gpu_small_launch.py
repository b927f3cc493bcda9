"""March launches around a task per warp and a task per CTA (each CTA's first block without the
queue, the queue after it) against the oracle bit for bit, over lists from the host and from the
device."""
import numpy as np
import pytest

from lum_gb300 import worldgen
from tests.helpers import random_prev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(20, 16, 16), (64, 64, 64)])   # staged in shared memory, and not
@pytest.mark.parametrize("n,rays", [(1, 32), (3, 32), (151, 32), (153, 32), (2432, 64), (2433, 64), (5000, 32), (1217, 128)])
def test_first_blocks(dims, n, rays):
    import lum_gb300
    import oracle
    w = worldgen.terrain_world(dims, seed=51)
    req = worldgen.all_probes(dims)[:n]
    prev = random_prev(w)
    with lum_gb300.RadianceWorld(dims, max_block_types=w.palette.shape[0]) as rw:
        rw.load(w)
        rw.set_radiance(prev)
        for seed in (0, 1):   # the queue is as the launch before left it
            rw.radiance_pass(req, lum_gb300.pass_params(rays=rays, max_dist=64.0, blend=0.1, time_seed=seed))
            prev, _, st = oracle.radiance_pass(w, req, prev=prev, rays=rays, max_dist=64.0, blend=0.1, time_seed=seed)
            got = rw.pass_stats()
            assert (got["steps"], got["hits"]) == (st["steps"], st["hits"])
        assert rw.get_radiance().tobytes() == prev.tobytes()


@pytest.mark.parametrize("block", [0, 3])
def test_device_list_shorter_than_the_launch(block):
    """update_radiance's list is read on the device: empty, and a few probes of a launch sized for all."""
    import lum_gb300
    import oracle
    w = worldgen.terrain_world((16, 12, 8), seed=52)
    w.grid = np.zeros_like(w.grid)
    w.grid[3, 4, 5] = block
    p = dict(rays=64, max_dist=64.0, blend=0.3, time_seed=2)
    prev = random_prev(w)
    with lum_gb300.RadianceWorld(w.dims, max_block_types=w.palette.shape[0]) as rw:
        rw.load(w)
        rw.set_radiance(prev)
        rw.update_radiance(lum_gb300.pass_params(**p))
        rw.update_radiance(lum_gb300.pass_params(**p))
        got = rw.get_radiance()
    for _ in range(2):
        prev, _, _ = oracle.radiance_pass(w, oracle.update_list(w), prev=prev, **p)
    assert got.tobytes() == prev.tobytes()
