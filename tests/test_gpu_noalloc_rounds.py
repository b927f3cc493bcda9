"""The no-allocation pass around the length of its rounds (4,096 subgroups), and over the world whose compact grid
leaves the least room for them, against the regular pass."""
import numpy as np
import pytest

from lum_gb300 import worldgen
from tests.helpers import RTOL, random_prev, rel_err
from tests.test_zz_no_alloc import _context_passes, _noalloc_passes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,rays,n", [((16, 16, 17), 32, 4088), ((16, 16, 17), 32, 4096), ((16, 16, 17), 32, 4097),
                                         ((9, 8, 8), 256, 512), ((9, 8, 8), 256, 513),
                                         ((1, 257, 2040), 32, 9000), ((1, 257, 2040), 128, 1100)])
def test_rounds(dims, rays, n):
    import lum_gb300
    w = worldgen.terrain_world(dims, seed=45, extra_blocks=dims[0] * dims[1])
    req = worldgen.all_probes(dims)
    at = np.r_[:n - n // 2, len(req) - n // 2:len(req)]   # the first and the last probes
    req = np.ascontiguousarray(req[at])
    prev = random_prev(w)
    params = [lum_gb300.pass_params(rays=rays, max_dist=96.0, blend=0.3, time_seed=s) for s in (2, 3)]
    want = _context_passes(w, req, prev, params)
    got = _noalloc_passes(w, req, prev, params)
    for i in range(2):
        assert rel_err(got[i], want[i]).max() <= RTOL
