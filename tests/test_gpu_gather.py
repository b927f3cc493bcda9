"""The gather's plain-point form against the oracle bit for bit: sizes around its CTAs, arrays that
are and are not 16-byte aligned, and points that take the general form (on a probe, not finite, far
away, huge normals, volumes with sums too small for the residual quotient)."""
import numpy as np
import pytest

from lum_gb300 import worldgen

pytestmark = pytest.mark.gpu


def _points(dims, n, seed):
    rng = np.random.default_rng(seed)
    pts = np.empty((n, 6), np.float32)
    pts[:, :3] = (rng.random((n, 3)) * 1.3 - 0.15) * np.array(dims) * 16
    nrm = rng.normal(size=(n, 3))
    pts[:, 3:] = nrm / np.linalg.norm(nrm, axis=1, keepdims=True)
    odd = [np.nan, np.inf, -np.inf, 1e30, -1e9, 0.0, -0.0, 8.0, 24.0, 8.0000005, 2.0 ** 61, 1e-30]
    k = rng.integers(0, n, 2 * len(odd))
    for i, v in enumerate(odd):
        pts[k[2 * i], rng.integers(0, 6)] = v
        pts[k[2 * i + 1], :3] = v
    return pts


@pytest.mark.parametrize("precision", ["fp32", "fp16", "bf16", "rgb10a2"])
@pytest.mark.parametrize("n", [1, 255, 256, 257, 5000])
@pytest.mark.parametrize("skew", [0, 1])
def test_gather_bits(precision, n, skew):
    import torch

    import lum_gb300
    import oracle
    dims = (9, 5, 3)
    w = worldgen.terrain_world(dims, seed=4)
    vol = (worldgen.uniform(5, 6, w.n_blocks * 3) * 1.0).astype(np.float32).reshape(w.grid.shape + (3,))
    vol[0, :3] = 0.0
    vol[1, :2] *= np.float32(1e-36)
    pts = _points(dims, n, 17 * n + skew)
    buf_p = torch.zeros(6 * n + 4, dtype=torch.float32, device="cuda")
    buf_o = torch.full((3 * n + 8,), -7.0, dtype=torch.float32, device="cuda")
    buf_p[skew:skew + 6 * n] = torch.from_numpy(pts.reshape(-1)).cuda()
    with lum_gb300.RadianceWorld(dims, max_block_types=w.palette.shape[0], precision=precision) as rw:
        rw.load(w)
        rw.set_radiance(vol)
        torch.cuda.synchronize()
        rw.gather_device(buf_p.data_ptr() + 4 * skew, n, buf_o.data_ptr() + 4 * skew)
        rw.synchronize()
        ref = oracle.gather(rw.get_radiance(), pts)
    got = buf_o.cpu().numpy()
    assert got[skew:skew + 3 * n].tobytes() == ref.tobytes()
    assert (got[:skew] == -7.0).all() and (got[skew + 3 * n:] == -7.0).all()   # nothing past the array
