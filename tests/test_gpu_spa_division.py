"""GPU test of the division in the flooding sum-product kernel.  Each of its four
call sites forms numerator and divisor from one float, so every operand pair that
can occur is tried: all floats of that value's range, compared bit for bit with
the correctly rounded __fdiv_rn (tolerance: none, the results are to be equal)."""
import ctypes
import os
import struct
import subprocess

import pytest

from gf2_b200 import build

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


def bits(x):
    return struct.unpack("<I", struct.pack("<f", x))[0]


@pytest.fixture(scope="module")
def lib(gpu, tmp_path_factory):
    out = str(tmp_path_factory.mktemp("spa_division") / "spa_division.so")
    subprocess.check_call([build.nvcc()] + build.flags() + ["-shared", "-I", build.CSRC, "-o", out,
                                                            os.path.join(HERE, "spa_division.cu")])
    lib = ctypes.CDLL(out)
    lib.spa_product_max.restype = ctypes.c_float
    return lib


@pytest.mark.parametrize("site", ["tanh", "atanh", "log", "log1p"])
def test_division_equals_fdiv_rn_for_every_operand_pair(lib, site):
    pmax = lib.spa_product_max()
    ranges = {"tanh": (0.0, 1.0), "atanh": (0.0, pmax), "log": (0.70710677, 1.4142137), "log1p": (0.0, 2.0 ** 25)}
    first, last = (bits(x) for x in ranges[site])
    out = (ctypes.c_ulonglong * 2)()
    assert lib.spa_division_check(list(ranges).index(site), first, last, out) == 0
    assert out[0] > (last - first) // 4 and out[1] == 0
