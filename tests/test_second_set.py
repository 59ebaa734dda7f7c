"""The second set of E and H of a closed box (whole-step kernel) is one allocation: it is
there whole or, when memory is short, not at all."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


def test_one_allocation(kh, gpu_lib, monkeypatch):
    from khronos_gb300.device import GpuSim

    sp = kh.Simulation(cell_size=(3.3, 2.1, 1.7), resolution=10, sources=[], dtype="f32").spec()

    def created():
        n0, n1, est, got = C.c_int64(), C.c_int64(), C.c_int64(), C.c_int64()
        assert gpu_lib.kh_device_alloc_count(C.byref(n0)) == 0
        g = GpuSim(sp, lib=gpu_lib)
        assert gpu_lib.kh_device_alloc_count(C.byref(n1)) == 0
        assert gpu_lib.kh_sim_memory_bytes(g.handle, C.byref(est), C.byref(got)) == 0
        g.close()
        return n1.value - n0.value, got.value

    created()  # whatever the first simulation of a process sets up
    with_set = created()
    monkeypatch.setenv("KHRONOS_GB300_FUSED", "0")
    without = created()
    assert with_set[0] - without[0] == 1
    assert with_set[1] > without[1]
