"""The march's regular-ray forms against the general ones, in FP32 on the CPU: for rays that start
in the world (probes at its borders and corners among them, direction components down to 2^-98)
every looked-up position is within one voxel of the world, the biased sums' bits give the general
form's cell, voxel and face, and no position is outside below the exit fraction."""
import numpy as np
import pytest

F = np.float32
BIAS = 2.0 ** 27


def rz_bits(q, bias, unit):
    """Bits of bias + q rounded toward zero to `unit` (the unit of bias's binade)."""
    s = np.floor((bias + q.astype(np.float64)) / unit) * unit
    return s.astype(F).view(np.uint32), s.astype(F)


def rays(rng, size, n):
    q = np.stack([rng.choice([0, s // 2, s - 1, int(rng.integers(s))], n) for s in size], axis=1)
    d = rng.normal(size=(n, 3))
    tiny = rng.random((n, 3)) < 0.25
    tiny[np.arange(n), rng.integers(0, 3, n)] = False
    d = np.where(tiny, np.sign(d) * 2.0 ** rng.uniform(-97, -3, (n, 3)), d)
    d = (d / np.sqrt((d * d).sum(1, keepdims=True))).astype(F)
    o = (q * 16 + 8).astype(F) + d * F(6)
    o = (o + (rng.random((n, 3)) - 0.5).astype(F) * F(2)).astype(F)
    flip = rng.random(n) < 0.5
    return o, np.where(flip[:, None], -d, d).astype(F)


@pytest.mark.parametrize("size", [(1, 1, 1), (2, 3, 1), (8, 8, 8), (45, 38, 11), (64, 64, 32), (2047, 5, 2047)])
def test_regular_forms_equal_general(size):
    rng = np.random.default_rng(sum(size))
    n = 6000
    o, d = rays(rng, size, n)
    iv = (F(1) / d).astype(F)
    assert np.isfinite(iv).all() and (np.abs(iv) <= F(2) ** 100 * F(1.001)).all()
    w = (np.array(size) * 16).astype(F)
    room = np.abs(np.where(d > 0, w, F(0)) - o).astype(F)
    fe = ((room - F(0.0078125)).astype(F) * np.abs(iv)).astype(F).min(1)
    fexit = np.maximum((fe * F(0.99999905)).astype(F), F(0))
    dims = np.array(size)
    px, py = size[0] + 1, size[1] + 1
    f = np.zeros(n, F)
    live = np.arange(n)
    outs = 0
    for _ in range(400 + 8 * max(size)):
        oo, dd, ii, fx = o[live], d[live], iv[live], fexit[live]
        f1 = (f[live] + F(0.5)).astype(F)
        p = (oo + (dd * f1[:, None]).astype(F)).astype(F)
        assert (p > -1).all() and (p < w + 1).all()
        # the general form's cell, voxel and face
        ip = np.trunc(p).astype(np.int64)
        cell = np.maximum(ip, 0) >> 4
        inside = ((ip >= -15) & (ip < 16 * dims)).all(1)
        face = (np.trunc((p * F(0.0625)).astype(F)) * F(16) + np.where(dd > 0, F(16), F(0))).astype(F)
        # the biased forms
        q = np.abs(p)
        tb, tv = rz_bits(q, BIAS, 16.0)
        idx = (tb[:, 0] + np.uint32(px) * (tb[:, 1] + np.uint32(py) * tb[:, 2])
               - np.uint32((0x4D000000 * (1 + px * (1 + py))) & 0xFFFFFFFF))
        want = cell[:, 0] + px * (cell[:, 1] + py * cell[:, 2])
        assert (idx.astype(np.int64) == want).all()
        assert ((cell <= dims).all(1)).all() and (inside | (cell == dims).any(1)).all()
        vx = rz_bits(q[:, 0], 2.0 ** 23, 1.0)[0] & 15
        vy = rz_bits(q[:, 1], 2.0 ** 22, 0.5)[0] & 0x1E
        vz = rz_bits(q[:, 2], 2.0 ** 18, 2.0 ** -5)[0] & 0x1E0
        v = ip & 15
        assert (vx == v[:, 0]).all() and (vy == 2 * v[:, 1]).all() and (vz == 32 * v[:, 2]).all()
        ahead = (tv + np.where(dd > 0, F(16 - BIAS), F(-BIAS))).astype(F)
        assert (ahead == face).all()
        t = ((face * ii).astype(F) - (p * ii).astype(F)).astype(F)
        skip = np.maximum(t.min(1), F(0.01))
        out = ((p < 0) | (p >= w)).any(1)
        assert (f1[out] >= fx[out]).all()
        outs += int(out.sum())
        air = rng.random(live.size) < 0.8
        f[live] = np.where(air, (f1 + skip).astype(F), f1)
        live = live[~out]
        if live.size == 0:
            break
    assert live.size < n // 50 and outs > n // 2
