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
int reduced(int nz, long long t, int s, int sms, int f64, int cpml) {
  return kh::reduced_zplanes(nz, t, s, sms, f64 != 0, cpml != 0);
}
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
    lib.reduced.argtypes = [C.c_int, C.c_longlong, C.c_int, C.c_int, C.c_int, C.c_int]
    return lib


SLOTS = 152 * 5


@pytest.mark.parametrize("n,want", [((64, 64, 64), 2), ((160, 160, 96), 7), ((256, 256, 128), 10),
                                    ((320, 192, 128), 10), ((256, 256, 256), 10), ((10, 10, 1), 1)])
def test_general_kernel_depth(plan, n, want):
    """Ten planes, or what fills two rounds of CTAs, whatever the precision."""
    assert plan.general(n[2], plan.tiles(n[0], n[1], 64, 4), SLOTS) == want


@pytest.mark.parametrize("nz", [65535, 65536, 131070, 131071, 300000, 458746, 655350, 4000000])
@pytest.mark.parametrize("f64", [0, 1])
def test_reduced_kernel_depth_within_the_launch_limits(plan, nz, f64):
    """At most 65535 CTAs along z, and at most the 64 planes a CTA has tables for."""
    z = plan.reduced(nz, 1, 152 * 3 if f64 else 152 * 6, 152, f64, 1)
    assert 1 <= z <= 64 and (nz + z - 1) // z <= 65535


@pytest.mark.parametrize("n,open_box,cpml", [((48, 48, 48), (2,), (2,)), ((64, 64, 64), (4,), (2, 3, 4)),
                                             ((100, 100, 100), (2, 3, 4, 6), (2, 3, 4, 6)),
                                             ((181, 97, 75), (2, 3, 4, 6), (2, 3, 4)),
                                             ((240, 144, 96), (2, 3, 4, 5, 6), (2, 3, 4, 5, 6)),
                                             ((320, 192, 128), (2, 3, 4, 5, 6), (2, 3, 4, 5, 6)),
                                             ((20, 20, 1), (1,), (1,))])
def test_fp64_depth(plan, n, open_box, cpml):
    """One of the depths measured within 8 % of the fastest (the figures beside the rule)."""
    t = plan.tiles(n[0], n[1], 64, 4)
    assert plan.reduced(n[2], t, 152 * 3, 152, 1, 0) in open_box
    assert plan.reduced(n[2], t, 152 * 3, 152, 1, 1) in cpml


@pytest.mark.gpu
def test_thin_column_above_the_launch_limits(kh, gpu_lib):
    """131080 planes: two planes a CTA (FP64) would be 65540 CTAs along z, and a thread
    block per plane 131080 in the export.  The exported state goes on bit for bit."""
    import numpy as np

    from khronos_gb300.device import GpuSim

    n = (2, 2, 131080)
    src = kh.UniformSource(time_profile=kh.GaussianPulseSource(fcen=0.8, fwidth=0.6), component=kh.EX,
                           center=(0, 0, 0), size=(0, 0, 0))
    sp = kh.Simulation(cell_size=tuple(a / 10 for a in n), resolution=10, sources=[src],
                       boundaries=[[0, 0], [0, 0], [0.5, 0.5]], dtype="f64").spec()
    assert tuple(sp.n) == n
    a, b = GpuSim(sp, lib=gpu_lib), GpuSim(sp, lib=gpu_lib)
    a.step(20)
    b.import_state(a.export_state())
    for g in (a, b):
        g.step(10)
        g.synchronize()
    assert np.any(a.field(kh.EX) != 0)
    assert np.array_equal(a.field(kh.EX), b.field(kh.EX))
    a.close()
    b.close()
