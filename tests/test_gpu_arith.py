"""The kernels' own reciprocal, square root and paired FP32 operations equal CUDA's correctly
rounded ones bit for bit: exhaustively over the mantissas of the ranges they are used in."""
import ctypes
import os
import subprocess

import pytest

from lum_gb300 import build

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("arith") / "arith_check.so")
    subprocess.run([build._nvcc(), *build.ARCH, *build.COMMON, *build.DEVICE, "-shared", "-cudart", "static",
                    os.path.join(HERE, "arith_check.cu"), "-o", so], check=True, capture_output=True)
    lib = ctypes.CDLL(so)
    lib.arith_check.restype = ctypes.c_longlong
    return lib.arith_check


@pytest.mark.gpu
@pytest.mark.parametrize("which", [0, 1, 2, 3], ids=["rcp", "sqrt", "pair_sum", "pair_difference"])
def test_bits_equal(check, which):
    assert check(which) == 0
