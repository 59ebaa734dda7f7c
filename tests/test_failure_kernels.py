"""Every kernel with shared-memory ring waits gives up on one that runs out, the host
learns of it, and the context stays usable: the whole-step kernel (a closed box), the
reduced-state kernel (an absorber) and the general kernel (CPU-path semantics), each in
the instantiation of the test hook whose first stage waits for bytes that are never sent."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("what,pml,launches", [("whole step", 0, 2), ("reduced state", 3, 4), ("general", 3, 4)])
@pytest.mark.parametrize("voxel", [False, True])
def test_timeout_is_reported_by_each_kernel(kh, gpu_lib, monkeypatch, what, pml, launches, voxel):
    from khronos_gb300 import _abi
    from khronos_gb300.device import GpuSim

    n = (70, 16, 12)
    sp = kh.Simulation(cell_size=tuple(a / 10 for a in n), resolution=10, sources=[],
                       boundaries=[[pml / 10, pml / 10]] * 3, dtype="f32").spec()
    assert tuple(sp.n) == n
    if voxel:
        for c in range(3):
            sp.materials.append((0, c, np.full(n, 0.5)))
    if what == "general":
        sp.semantics = 0
    monkeypatch.setenv("KHRONOS_GB300_GRAPHS", "0")
    monkeypatch.setenv("KHRONOS_GB300_TEST_STALL", "1")
    g = GpuSim(sp, lib=gpu_lib)
    monkeypatch.delenv("KHRONOS_GB300_TEST_STALL")
    before = g.launches
    with pytest.raises(_abi.KhError) as e:
        g.step(2)
        g.synchronize()
    assert e.value.status == _abi.KH_ERR_TIMEOUT
    assert g.launches - before == launches
    g.close()

    ok = GpuSim(sp, lib=gpu_lib)
    ok.step(20)
    ok.synchronize()
    ok.check_finite()
    ok.close()
