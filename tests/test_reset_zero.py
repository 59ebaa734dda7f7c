"""reset() zeroes the state arrays together: more of them than one launch takes, and
DFT arrays whose length is no multiple of 16 bytes or of a block's piece."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["f32", "f64"])
@pytest.mark.parametrize("count", [1, 5, 75])
def test_reset_zeroes_everything(kh, gpu_lib, dtype, count):
    from khronos_gb300.device import GpuSim
    from khronos_gb300.spec import MonitorSpec

    src = kh.UniformSource(time_profile=kh.GaussianPulseSource(fcen=0.8, fwidth=0.4), component=kh.EZ,
                           center=(0, 0, 0), size=(0, 0, 0))
    sp = kh.Simulation(cell_size=(3.3, 2.9, 2.7), resolution=10, sources=[src], boundaries=[[0.4, 0.4]] * 3,
                       dtype=dtype).spec()
    boxes = [(1, 1, 1), (3, 5, 7), (1, 29, 27), (33, 7, 9), (16, 16, 8)]
    for m in range(count):
        sp.monitors.append(MonitorSpec(component=m % 6, start=(0, 0, 0), dims=boxes[m % 5],
                                       freqs=np.linspace(0.7, 0.9, 1 + m % 3), decimation=1))
    g = GpuSim(sp, lib=gpu_lib)
    g.step(60)
    ref = [g.field(c) for c in range(6)] + [g.dft(m) for m in range(count)]
    assert any(np.any(a != 0) for a in ref)
    g.reset()
    assert g.timestep == 0
    assert not any(np.any(a != 0) for a in [g.field(c) for c in range(6)] + [g.dft(m) for m in range(count)])
    assert not any(g.export_state()[16:])
    g.step(60)
    for a, b in zip(ref, [g.field(c) for c in range(6)] + [g.dft(m) for m in range(count)]):
        assert np.array_equal(a, b)
    g.close()
