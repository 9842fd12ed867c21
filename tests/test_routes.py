"""The rules that pick a kernel by sizes (csrc/it_route.h), held to their edges on the CPU.  148 SMs are a B200's."""
import ctypes as C
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "irontimber_b200", "csrc")
SM = 148


@pytest.fixture(scope="module")
def routes(tmp_path_factory):
    d = tmp_path_factory.mktemp("routes")
    src, lib = d / "routes.cpp", d / "routes.so"
    src.write_text('#include "it_route.h"\n'
                   'extern "C" int takes_tc(long rg, long ntok, int sm) { return it_mm_takes_tc(rg, ntok, sm); }\n')
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-Wno-unused-function", "-shared", "-fPIC", "-I", CSRC, str(src), "-o", str(lib)], check=True)
    return C.CDLL(str(lib))


@pytest.mark.parametrize("rows,ntok,tc", [
    (5120, 32, 0), (5120, 40, 0), (5120, 41, 1), (5120, 64, 1), (5120, 65, 1), (5120, 128, 1), (5120, 236, 1),      # one wave and twelve CTAs of 32-row tiles
    (4736, 64, 0), (4737, 64, 1), (4736, 65, 0), (2560, 64, 0), (1024, 512, 0),                                     # no more row groups than SMs
    (5568, 40, 0), (5569, 40, 1), (5569, 32, 0), (6144, 32, 0), (6144, 33, 1), (11136, 33, 1),                       # from 5569 on: 64-row tiles
    (11137, 9, 1), (34816, 9, 1), (2689, 256, 1), (2688, 256, 0)])                                  # 128-row tiles for 0.6 of the SMs
def test_tile_kernel_of_a_product(routes, rows, ntok, tc):
    assert routes.takes_tc(C.c_long((rows + 31) // 32), C.c_long(ntok), SM) == tc
