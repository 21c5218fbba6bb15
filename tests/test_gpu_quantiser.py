"""The q8_1 quantiser's division by 127 and its rounding of a code, against the operations that they replace: every mantissa at
the exponents where something changes (the smallest amax that counts, where the remainder is nearly subnormal; the middle; the
largest finite values and infinity), and every float that can become a code, ties included, and NaN."""
import ctypes
import os
import subprocess

import pytest

from bonsai_vk_b200.build import NVCC_FLAGS

pytestmark = pytest.mark.gpu
SRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "native", "quant_check.cu")


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("native") / "quant_check.so")
    subprocess.run(["nvcc", *NVCC_FLAGS, "-o", so, SRC], check=True, capture_output=True, timeout=300)
    lib = ctypes.CDLL(so)
    lib.check_div127.restype = lib.check_code_byte.restype = ctypes.c_longlong
    lib.check_div127.argtypes = [ctypes.c_uint]
    lib.check_code_byte.argtypes = [ctypes.c_uint, ctypes.c_uint]
    return lib


@pytest.mark.parametrize("exponent", [10, 11, 12, 13, 17, 18, 24, 64, 126, 127, 128, 133, 200, 253, 254])
def test_division_by_127(probe, exponent):
    assert probe.check_div127(exponent) == 0


def test_division_of_infinity(probe):
    # exponent 255: infinity divides to itself; a NaN amax does not occur (a maximum leaves NaNs out, and x > 1e-35 is false)
    assert probe.check_div127(255) == 0


@pytest.mark.parametrize("first,last", [(0x00000000, 0x42FEFFFF), (0x80000000, 0xC2FF0000), (0x7FC00000, 0x7FC00000), (0xFFC00000, 0xFFC00000)])
def test_codes(probe, first, last):
    """0 .. below 127.5, -0 .. -127.5, NaN of either sign."""
    assert probe.check_code_byte(first, last - first + 1) == 0
