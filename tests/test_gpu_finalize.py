"""Passes without hit records (the packed finalize, regular and irregular rays) against the oracle bit
for bit: launches of few and of many groups, lists that end inside a group, ray counts whose
subgroups do and do not share a CTA, probes outside the world (their rays are not regular), voxels in
block 0 (hits in air and past the world's far faces) and block ids without a palette slot."""
import numpy as np
import pytest

from lum_gb300 import worldgen
from tests.helpers import random_prev

pytestmark = pytest.mark.gpu


def _run(w, req, **p):
    import lum_gb300
    import oracle
    prev = random_prev(w)
    with lum_gb300.RadianceWorld(w.dims, max_block_types=w.palette.shape[0]) as rw:
        rw.load(w)
        rw.set_radiance(prev)
        rw.radiance_pass(req, lum_gb300.pass_params(**p))
        got, st = rw.get_radiance(), rw.pass_stats()
    ref, _, rst = oracle.radiance_pass(w, req, prev=prev, **p)
    assert (st["steps"], st["hits"], st["rays"]) == (rst["steps"], rst["hits"], rst["rays"])
    assert got.tobytes() == ref.tobytes()


@pytest.mark.parametrize("dims,rays", [((12, 10, 7), 32), ((44, 40, 12), 64), ((45, 31, 9), 96), ((12, 11, 6), 96),
                                       ((24, 20, 9), 160), ((33, 30, 11), 256), ((9, 7, 5), 1024)])
def test_pass_bits(dims, rays):
    w = worldgen.terrain_world(dims, seed=41, extra_blocks=dims[0] * dims[1])
    req = worldgen.all_probes(dims)[:-3]
    _run(w, req, rays=rays, max_dist=128.0, blend=0.1, time_seed=9)


@pytest.mark.parametrize("dims,size,shift", [((11, 9, 6), 1, 0), ((11, 9, 6), 3, 2), ((48, 44, 11), 1, 0)])
def test_odd_worlds(dims, size, shift):
    w = worldgen.terrain_world(dims, seed=42, extra_blocks=60)
    w.palette[0] = (worldgen.uniform(1, 2, 4096) < 0.002).reshape(16, 16, 16) * 5   # voxels in "air"
    g = w.grid.reshape(-1)
    g[worldgen.randint(3, 4, 30, 0, g.size)] = -worldgen.randint(5, 6, 30, 1, 70).astype(np.int16)
    g[worldgen.randint(7, 8, 10, 0, g.size)] = 900
    req = worldgen.all_probes(dims)
    X, Y, Z = dims
    outside = np.array([[-1, 2, 2, 0], [X, 3, 3, 0], [4, -2, 1, 0], [4, Y, 1, 0], [5, 5, Z, 0], [5, 5, -1, 0],
                        [-300, 7, 2, 0], [30000, -30000, 12, 0]], np.int16)
    req = np.concatenate([req[:50], outside[:4], req[50:], outside[4:]])
    _run(w, req, rays=64, max_dist=96.0, blend=0.2, time_seed=3, size=size, shift=shift)
