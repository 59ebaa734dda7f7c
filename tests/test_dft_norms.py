"""kh_sim_dft_norms with every monitor of a batch in one launch: norms of the arrays
that kh_sim_read_dft returns, for monitors around a block's chunk (4096 values) and
for more monitors than one batch holds.  Both are FP64 sums of n squares of the same
values, in another order: relative difference at most n·2^-53."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["f32", "f64"])
@pytest.mark.parametrize("count", [1, 32, 33, 70])
def test_norms_match_the_arrays(kh, gpu_lib, dtype, count):
    from khronos_gb300.device import GpuSim
    from khronos_gb300.spec import MonitorSpec

    src = kh.UniformSource(time_profile=kh.GaussianPulseSource(fcen=0.8, fwidth=0.4), component=kh.EZ,
                           center=(0, 0, 0), size=(0, 0, 0))
    sp = kh.Simulation(cell_size=(3.6, 3.4, 3.4), resolution=10, sources=[src], dtype=dtype).spec()
    boxes = [(1, 1, 1), (1, 32, 32), (32, 32, 4), (33, 31, 4), (16, 16, 16), (17, 16, 16)]
    for m in range(count):
        sp.monitors.append(MonitorSpec(component=m % 6, start=(1, 1, 1), dims=boxes[m % len(boxes)],
                                       freqs=np.linspace(0.7, 0.9, 1 + m % 4), decimation=1))
    g = GpuSim(sp, lib=gpu_lib)
    g.step(50)
    got = g.dft_norms()
    assert got.shape == (count,)
    for m in range(count):
        d = g.dft(m)
        want = np.sqrt(np.sum(d.real ** 2 + d.imag ** 2))
        assert abs(got[m] - want) <= max(4, d.size) * 2.0 ** -53 * want
    g.close()
