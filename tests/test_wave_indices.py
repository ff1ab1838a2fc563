"""Where the threads of a wavefront sweep read, on the CPU: the kernel's index arithmetic
(csrc/wave_place.hpp) evaluated for every thread of every tile in all four sweeps. Threads
without a pencil (ny or nz no multiple of the tile) stay inside the arrays like the others."""
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
    out = str(tmp_path_factory.mktemp("wave") / "libwave_harness.so")
    subprocess.run([cxx, "-O1", "-std=c++17", "-fPIC", "-shared", "-I", SRC, "-o", out,
                    os.path.join(HERE, "native", "wave_harness.cpp")], check=True, capture_output=True)
    return C.CDLL(out)


@pytest.mark.parametrize("mode", ["ic0 forward", "ic0 backward", "gauss-seidel forward", "gauss-seidel backward"])
@pytest.mark.parametrize("cells", [(2, 9, 7), (3, 8, 8), (17, 17, 9), (300, 5, 3), (21, 24, 16), (2, 2, 2), (24, 20, 16),
                                   (75, 61, 37), (100, 92, 50), (5, 33, 1000)])
def test_every_read_is_inside_the_arrays(harness, cells, mode):
    modes = ["ic0 forward", "ic0 backward", "gauss-seidel forward", "gauss-seidel backward"]
    out = (C.c_int64 * 4)()
    harness.wave_scan(modes.index(mode), *cells, out)
    assert out[3] > 0
    assert (out[0], out[1], out[2]) == (0, 0, 0)
