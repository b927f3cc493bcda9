"""The block and compact-grid cells that the kernels look up (csrc/lumrad_cells.h, compiled for the host), up to the
largest accepted worlds: their compact grids have more than 2^31 cells."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lum_gb300", "csrc")

SRC = r"""
#include "lumrad_cells.h"
using namespace lumrad;
// the element `idx` names, as a load through it forms the address (from the array's start)
extern "C" int cells(const int* dims, int pad, const int* voxel, long long* at, unsigned long long* n) {
    static const char* base = 0;
    auto idx = cell_index(1, 1, 0, 0, 0);
    const bool in = grid_index(dims[0], dims[1], dims[2], dims[0] + pad, dims[1] + pad, voxel[0], voxel[1], voxel[2], idx);
    *at = (long long)((unsigned long long)(base + idx) - (unsigned long long)base);
    *n = compact_cells(dims[0], dims[1], dims[2]);
    return in;
}
extern "C" long long cell(const int* dims, const int* b) {
    static const char* base = 0;
    return (long long)((unsigned long long)(base + cell_index(dims[0] + 1, dims[1] + 1, b[0], b[1], b[2])) - (unsigned long long)base);
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("cells")
    src, out = d / "cells.cpp", d / "cells.so"
    src.write_text(SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, str(src), "-o", str(out)], check=True)
    so = C.CDLL(str(out))
    so.cell.restype = C.c_longlong
    return so


@pytest.mark.parametrize("dims", [(1, 1, 1), (64, 64, 16), (2047, 3, 2), (2047, 2047, 512), (512, 2047, 2047), (1290, 1290, 1290)])
def test_cells(lib, dims):
    X, Y, Z = dims
    assert X * Y * Z < 2 ** 31
    d = (C.c_int * 3)(*dims)
    at, n = C.c_longlong(), C.c_ulonglong()
    rng = np.random.default_rng(X)
    voxels = [(16 * X - 1, 16 * Y - 1, 16 * Z - 1), (0, 0, 0), (-15, -1, -15), (16 * X - 1, 0, 16 * Z - 16), (-16, 0, 0),
              (16 * X, 16 * Y, 16 * Z), (0, 16 * Y - 1, 16 * Z - 1), (2 ** 31 - 1, -2 ** 31, 5)]
    voxels += [tuple(int(t) for t in rng.integers(-20, 16 * np.array(dims) + 20)) for _ in range(200)]
    for v in voxels:
        want_in = all(-15 <= t < 16 * s for t, s in zip(v, dims))
        bx, by, bz = (max(t, 0) >> 4 for t in v)
        for pad in (0, 1):   # the grid, the compact grid
            got_in = lib.cells(d, pad, (C.c_int * 3)(*v), C.byref(at), C.byref(n))
            assert bool(got_in) == want_in
            if want_in:
                assert at.value == bx + (X + pad) * (by + (Y + pad) * bz)
        assert n.value == (X + 1) * (Y + 1) * (Z + 1)
    # the cells one past the grid, which the regular rays' lookups read without a range test
    for b in ((X, Y, Z), (X, 0, 0), (X - 1, Y, Z), (0, 0, Z), (X, Y - 1, Z - 1)):
        want = b[0] + (X + 1) * (b[1] + (Y + 1) * b[2])
        assert lib.cell(d, (C.c_int * 3)(*b)) == want < n.value
