"""The device's dirty list on both sides of each line between its two forms (edits, rows, list length), at worlds' faces and
with cubes larger than the world on an axis, against the host's list."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# edits 4,096 | 4,097; rows (of 8x8 inside 8x8x8) 131,072 | 131,136; list bound (125 an edit) 65,536; an axis of one block
@pytest.mark.parametrize("dims,n,radius", [((64, 64, 16), 4096, 0), ((64, 64, 16), 4097, 0), ((8, 8, 8), 2048, 5), ((8, 8, 8), 2049, 5),
                                           ((64, 64, 64), 524, 2), ((64, 64, 64), 525, 2), ((1, 40, 3), 50, 15), ((2047, 1, 2), 9, 15),
                                           ((5, 1, 90), 30, 4)])
@pytest.mark.parametrize("kind", ["faces", "same", "spread"])
def test_dirty_line(dims, n, radius, kind):
    import lum_gb300
    rng = np.random.default_rng(n + radius)
    edits = np.zeros((n, 4), np.int16)
    for a in range(3):
        edits[:, a] = {"faces": rng.choice([0, dims[a] - 1], n), "same": np.full(n, dims[a] // 2),
                       "spread": rng.integers(0, dims[a], n)}[kind]
    with lum_gb300.RadianceWorld(dims, max_block_types=4) as rw:
        assert np.array_equal(rw.build_dirty_list(edits, radius), lum_gb300.dirty_probes(dims, edits, radius))
