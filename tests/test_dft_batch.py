"""Batched DFT accumulation at the sizes where its dispatch changes: one item per
thread in small launches, eight frequencies and two cells above, one cell per
thread for a monitor with an odd number of cells.  The one-monitor kernel
(KHRONOS_GB300_DFT_BATCH=0) does the same additions, so the bar is equality."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["f32", "f64"])
@pytest.mark.parametrize("dims,nf", [((1, 1, 1), 1), ((5, 7, 3), 3), ((1, 33, 31), 21), ((48, 41, 2), 9),
                                     ((1, 160, 160), 17), ((161, 1, 161), 16), ((40, 40, 40), 8)])
def test_batched_equals_single(kh, gpu_lib, monkeypatch, dtype, dims, nf):
    from khronos_gb300.device import GpuSim
    from khronos_gb300.spec import MonitorSpec

    n = tuple(max(24, d + 3) for d in dims)
    src = kh.UniformSource(time_profile=kh.GaussianPulseSource(fcen=0.8, fwidth=0.4), component=kh.EZ,
                           center=(0, 0, 0), size=(0, 0, 0))
    sp = kh.Simulation(cell_size=tuple(a / 10 for a in n), resolution=10, sources=[src], dtype=dtype).spec()
    assert tuple(sp.n) == n
    for comp in (kh.EZ, kh.HX, kh.EY):
        sp.monitors.append(MonitorSpec(component=comp, start=(1, 2, 1), dims=dims,
                                       freqs=np.linspace(0.6, 1.0, nf), decimation=1))
    out = []
    for mode in ("0", "1"):
        monkeypatch.setenv("KHRONOS_GB300_DFT_BATCH", mode)
        g = GpuSim(sp, lib=gpu_lib)
        g.step(60)
        out.append([g.dft(m) for m in range(3)])
        g.close()
    assert dims == (1, 1, 1) or any(np.any(d != 0) for d in out[0])
    for a, b in zip(*out):
        assert np.array_equal(a, b)
