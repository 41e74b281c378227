"""Where a node's values lie (csrc/e3d_index.h) on grids of more than 2^30 nodes, which
batched and served solves may have: no device in these tests holds one, so the
arithmetic that the kernels share is checked on the host."""
import ctypes as C
import os
import subprocess

import pytest

import elas3d_xtal_gb300 as e3d

CSRC = os.path.join(os.path.dirname(os.path.abspath(e3d.__file__)), "csrc")
SOURCE = """
#include "e3d_index.h"
extern "C" unsigned node(unsigned col, unsigned nxy, int z) { return e3d::node_of(col, nxy, z); }
extern "C" unsigned long long bytes4(unsigned m) { return e3d::node_bytes4(m); }
extern "C" unsigned long long value(unsigned m, int c, long long ns) { return e3d::value_of(m, c, ns); }
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("index")
    (d / "i.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, str(d / "i.cpp"), "-o", str(d / "i.so")],
                   check=True)
    lib = C.CDLL(str(d / "i.so"))
    lib.node.argtypes, lib.node.restype = [C.c_uint, C.c_uint, C.c_int], C.c_uint
    lib.bytes4.argtypes, lib.bytes4.restype = [C.c_uint], C.c_ulonglong
    lib.value.argtypes, lib.value.restype = [C.c_uint, C.c_int, C.c_longlong], C.c_ulonglong
    return lib


@pytest.mark.parametrize("shape", [(64, 8, 33), (1024, 1024, 1024), (1025, 1024, 1024), (1040, 1040, 1040),
                                   (1100, 1100, 1100), (36000, 36000, 1), (1, 36000, 36000)])
def test_offsets(lib, shape):
    nx, ny, nz = shape
    ns = nx * ny * nz
    assert ns < 2 ** 32
    for x in {0, nx // 2, nx - 1}:
        for y in {0, ny // 2, ny - 1}:
            for z in {0, nz // 2, nz - 1}:
                m = lib.node(x + nx * y, nx * ny, z)
                assert m == x + nx * (y + ny * z)
                assert lib.bytes4(m) == 4 * m
                for c in range(6):  # six values of an inverse block
                    assert lib.value(m, c, ns) == m + c * ns
