"""The list builders around their CTA edges and past the size up to which a CTA sums the counts before
it, with and without specials, against the oracle and the host's list; and frames back to back (each
frame's launches start in the tail of the one before) against the same passes one by one."""
import numpy as np
import pytest

from lum_gb300 import worldgen
from tests.helpers import random_prev

pytestmark = pytest.mark.gpu


def _world(dims, seed):
    w = worldgen.terrain_world(dims, seed=seed)
    g = w.grid.reshape(-1)
    k = worldgen.randint(seed, 5, max(1, g.size // 40), 0, g.size)
    g[k] = -worldgen.randint(seed, 6, k.size, 0, 20).astype(np.int16)
    return w


@pytest.mark.parametrize("dims", [(255, 1, 1), (16, 16, 1), (257, 1, 1), (3, 7, 61), (128, 128, 66)])
@pytest.mark.parametrize("specials", [False, True])
def test_lists(dims, specials):
    import lum_gb300
    import oracle
    w = _world(dims, 61)
    sp = np.array([[0, 0, 0, 0], [dims[0] - 1, dims[1] - 1, dims[2] - 1, 0], [dims[0] // 2, 0, dims[2] - 1, 0]], np.int16)
    with lum_gb300.RadianceWorld(dims, max_block_types=w.palette.shape[0]) as rw:
        rw.load(w)
        if specials:
            for s in sp:
                rw.request_update(*[int(v) for v in s[:3]])
        got = rw.build_update_list()
        ref = oracle.update_list(w, sp) if specials else oracle.update_list(w)
        assert np.array_equal(got, ref)
        edits = worldgen.edit_request(dims, 0.002, seed=3, stream=0)
        for radius in (0, 2):
            assert np.array_equal(rw.build_dirty_list(edits, radius), lum_gb300.dirty_probes(dims, edits, radius))


@pytest.mark.parametrize("dims", [(8, 8, 8), (45, 38, 11)])
def test_frames_back_to_back(dims):
    import torch

    import lum_gb300
    w = _world(dims, 62)
    prev = random_prev(w)
    pts = np.random.default_rng(1).random((3000, 6)).astype(np.float32) * 60
    p = [lum_gb300.pass_params(rays=64, max_dist=64.0, blend=0.3, time_seed=k) for k in range(12)]
    d_pts = torch.from_numpy(pts).cuda()
    outs = torch.zeros((12, 3000, 3), dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    with lum_gb300.RadianceWorld(dims, max_block_types=w.palette.shape[0]) as a, \
            lum_gb300.RadianceWorld(dims, max_block_types=w.palette.shape[0]) as b:
        for rw in (a, b):
            rw.load(w)
            rw.set_radiance(prev)
        a.set_radiance_shift(1, 0, 0)
        for k in range(12):
            a.update_radiance(p[k])
            a.gather_device(d_pts.data_ptr(), 3000, outs[k].data_ptr())
        a.synchronize()
        req = b.build_update_list()
        for k in range(12):
            b.shift_radiance(1, 0, 0)
            b.synchronize()
            b.radiance_pass(req, p[k])
            assert b.gather(pts).tobytes() == outs[k].cpu().numpy().tobytes()
        assert a.get_radiance().tobytes() == b.get_radiance().tobytes()


@pytest.mark.parametrize("dims", [(31, 9, 5), (64, 64, 64), (2047, 3, 2), (65, 64, 64)])
@pytest.mark.parametrize("n,radius", [(0, 2), (1, 0), (1, 15), (700, 3), (2200, 15)])
def test_dirty_lists(dims, n, radius):
    """Both forms of the dirty list (rows of bits; the dilation of larger worlds and edit counts)."""
    import lum_gb300
    rng = np.random.default_rng(n + radius)
    edits = np.zeros((n, 4), np.int16)
    for a in range(3):
        edits[:, a] = rng.choice([0, dims[a] - 1, dims[a] // 2, -1], n) if n else 0
        wild = edits[:, a] < 0
        edits[wild, a] = rng.integers(0, dims[a], int(wild.sum()))
    with lum_gb300.RadianceWorld(dims, max_block_types=4) as rw:
        for _ in range(2):
            assert np.array_equal(rw.build_dirty_list(edits, radius), lum_gb300.dirty_probes(dims, edits, radius))
