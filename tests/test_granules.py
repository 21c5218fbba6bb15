"""Where the single projection reads native rows of 4-byte alignment: the kernel's own arithmetic, compiled for the host, over every tile,
group and lane - no byte outside of the matrix, every byte of the rows at the place where the kernel looks for it - for every place of
the matrix in a granule, heights around one and several tiles and block counts around the groups of four."""
import ctypes
import os
import subprocess

import pytest

SRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "native", "granule_check.cpp")


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("native") / "granule_check.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-Wall", "-Wno-unknown-pragmas", "-shared", "-fPIC", "-o", so, SRC], check=True, timeout=120)
    f = ctypes.CDLL(so).check_granules
    f.restype, f.argtypes = ctypes.c_longlong, [ctypes.c_ulonglong, ctypes.c_int, ctypes.c_int]
    return f


@pytest.mark.parametrize("nb", [1, 2, 3, 4, 5, 6, 7, 9, 13, 37])
def test_copies_stay_in_the_matrix_and_bring_it_all(check, nb):
    for M in (1, 2, 15, 16, 17, 18, 19, 20, 31, 32, 33, 34, 36, 47, 48, 49, 113):
        for place in (0, 4, 8, 12):
            assert check(0x7000000 + place, M, nb) == 0, f"{M} rows at {place}"
