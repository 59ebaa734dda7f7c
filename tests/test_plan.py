"""How the step kernels split a grid (csrc/kh_plan.h), compiled for the host."""
import ctypes as C
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "khronos.jl_gb300" / "csrc"
WRAP = """
#include "kh_plan.h"
extern "C" {
long long tiles(int nx, int ny, int tx, int ty) { return kh::plan_tiles(nx, ny, tx, ty); }
int general(int nz, long long t, int s) { return kh::general_zplanes(nz, t, s); }
int reduced(int nz, long long t, int s, int f64) { return kh::reduced_zplanes(nz, t, s, f64 != 0); }
}
"""


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    (d / "wrap.cpp").write_text(WRAP)
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-shared", "-fPIC", "-I", str(CSRC),
                    str(d / "wrap.cpp"), "-o", str(d / "plan.so")], check=True)
    lib = C.CDLL(str(d / "plan.so"))
    lib.tiles.restype = C.c_longlong
    lib.general.argtypes = [C.c_int, C.c_longlong, C.c_int]
    lib.reduced.argtypes = [C.c_int, C.c_longlong, C.c_int, C.c_int]
    return lib


SLOTS = 152 * 5


@pytest.mark.parametrize("n,want", [((64, 64, 64), 2), ((160, 160, 96), 7), ((256, 256, 128), 10),
                                    ((320, 192, 128), 10), ((256, 256, 256), 10), ((10, 10, 1), 1)])
def test_general_kernel_depth(plan, n, want):
    """Ten planes, or what fills two rounds of CTAs, whatever the precision."""
    assert plan.general(n[2], plan.tiles(n[0], n[1], 64, 4), SLOTS) == want
