"""Passes with hit records around the line between the finalize's two widths (launches of few groups run a warp per
task), in the lean and the general form: records and volume bit for bit those of the oracle."""
import pytest

from lum_gb300 import worldgen
from tests.helpers import oracle_pass, random_prev

pytestmark = pytest.mark.gpu

FEW = 16    # groups of eight tasks per SM


@pytest.mark.parametrize("rays", [32, 64, 96, 256])
@pytest.mark.parametrize("extra", [0, 1])   # the last launch of few groups, the first of many
def test_records_at_the_line(rays, extra):
    import torch

    import lum_gb300
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    dims = (40, 36, 14)
    w = worldgen.terrain_world(dims, seed=43, extra_blocks=900)
    n = FEW * sms * 8 * 32 // rays + extra
    req = worldgen.all_probes(dims)[:n]
    assert len(req) == n
    prev = random_prev(w)
    p = dict(rays=rays, max_dist=96.0, blend=0.2, time_seed=5)
    with lum_gb300.RadianceWorld(dims, max_block_types=w.palette.shape[0]) as rw:
        rw.load(w)
        rw.set_radiance(prev)
        rw.radiance_pass(req, lum_gb300.pass_params(record_hits=True, **p))
        got, hits, st = rw.get_radiance(), rw.get_hits(), rw.pass_stats()
    ref, ref_hits, rst = oracle_pass(w, req, prev, **p)
    assert hits.tobytes() == ref_hits.tobytes()
    assert got.tobytes() == ref.tobytes()
    assert (st["steps"], st["hits"]) == (rst["steps"], rst["hits"])
