"""lumrad_get_radiance into page-locked and pageable arrays, aligned and not, whole allocations and
parts of them: the same volume, and nothing written past it."""
import numpy as np
import pytest

from lum_gb300 import worldgen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32", "fp16", "bf16", "rgb10a2"])
@pytest.mark.parametrize("dims", [(1, 1, 1), (8, 8, 4), (17, 5, 3), (33, 31, 9)])
@pytest.mark.parametrize("pinned,skew", [(True, 0), (True, 1), (True, 4), (False, 0)])
def test_readback(precision, dims, pinned, skew):
    import torch

    import lum_gb300
    n = 3 * dims[0] * dims[1] * dims[2]
    vol = worldgen.uniform(7, 8, n).astype(np.float32).reshape(dims[::-1] + (3,))
    buf = torch.full((n + skew + 5,), -3.0, dtype=torch.float32, pin_memory=pinned).numpy()
    with lum_gb300.RadianceWorld(dims, max_block_types=4, precision=precision) as rw:
        rw.set_radiance(vol)
        plain = rw.get_radiance()
        rw.get_radiance(buf[skew:skew + n])
    tol = {"fp32": 0.0, "fp16": 2.0 ** -11, "bf16": 2.0 ** -8, "rgb10a2": 0.5 / 1023 + 1e-7}[precision]
    assert np.abs(plain - vol).max() <= tol   # the storage type's rounding of values below 1
    assert buf[skew:skew + n].tobytes() == plain.tobytes()
    assert (buf[:skew] == -3.0).all() and (buf[skew + n:] == -3.0).all()
