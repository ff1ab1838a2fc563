"""The slots of a bin level taken apart through products (csrc/bin_div.hpp), on the CPU: every
quotient of every level that is accepted for it, and levels with wrong quotients that are not."""
import ctypes as C
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(os.path.dirname(HERE), "cfd-craft_gb300", "csrc")


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no C++ compiler")
    out = str(tmp_path_factory.mktemp("bins") / "libbin_harness.so")
    subprocess.run([cxx, "-O2", "-std=c++17", "-fPIC", "-shared", "-I", SRC, "-o", out,
                    os.path.join(HERE, "native", "bin_harness.cpp")], check=True, capture_output=True)
    lib = C.CDLL(out)
    lib.bin_scan.restype = C.c_int64
    lib.bin_scan.argtypes = lib.bin_exact.argtypes = [C.c_int64, C.c_int, C.c_int]
    return lib


# Bins per row and colour, bin rows per layer, layers.
@pytest.mark.parametrize("nbh, nby, nbz", [(1, 1, 9), (1, 3, 5), (4, 7, 1), (32, 64, 32), (25, 42, 25), (3, 10921, 11),
                                           (1, 32767, 3), (4, 2047, 500), (32767, 1, 3), (7, 4681, 27)])
def test_accepted_levels_are_exact(harness, nbh, nby, nbz):
    rows = nbh * nby * nbz
    assert harness.bin_exact(rows, nbh, nby)
    assert harness.bin_scan(rows, nbh, nby) == 0


@pytest.mark.parametrize("nbh, nby, nbz", [(1, 32766, 6), (2, 16381, 41), (4, 4093, 700)])
def test_levels_with_wrong_quotients_are_refused(harness, nbh, nby, nbz):
    """Few bins in x and many in y: the products with nbh alone are in range."""
    rows = nbh * nby * nbz
    assert rows * nbh < 1 << 32
    assert harness.bin_scan(rows, nbh, nby) > 0
    assert not harness.bin_exact(rows, nbh, nby)
