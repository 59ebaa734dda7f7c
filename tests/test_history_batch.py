"""History monitors recorded together: more of them than one launch holds, both halves'
components, boxes of one cell, of one row, wider than a block and with many rows, some
whose capacity ends early.  Copies: the bar is equality with the fields."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["f32", "f64"])
def test_records_equal_fields(kh, gpu_lib, dtype):
    from khronos_gb300.device import GpuSim
    from khronos_gb300.spec import HistorySpec

    src = kh.UniformSource(time_profile=kh.GaussianPulseSource(fcen=0.8, fwidth=0.4), component=kh.EZ,
                           center=(0, 0, 0), size=(0, 0, 0))
    sp = kh.Simulation(cell_size=(7.0, 2.3, 2.1), resolution=10, sources=[src], boundaries=[[0.4, 0.4]] * 3,
                       dtype=dtype).spec()
    boxes = [((3, 2, 1), (1, 1, 1)), ((0, 0, 0), (70, 23, 21)), ((5, 7, 4), (33, 1, 1)), ((1, 0, 3), (1, 23, 17)),
             ((2, 3, 3), (64, 5, 2)), ((0, 11, 10), (70, 1, 9)), ((30, 1, 1), (7, 20, 3))]
    for q in range(29):
        st, dm = boxes[q % len(boxes)]
        sp.histories.append(HistorySpec(component=q % 6, start=st, dims=dm, capacity=6 if q % 4 == 3 else 12))
    g = GpuSim(sp, lib=gpu_lib)
    seen = False
    for t in range(9):
        g.step(1)
        f = [g.field(c) for c in range(6)]
        for q, h in enumerate(sp.histories):
            if t >= h.capacity:
                continue
            box = tuple(slice(h.start[a], h.start[a] + h.dims[a]) for a in range(3))
            got = g.history(q, t)
            assert np.array_equal(got, f[h.component][box]), (t, q)
            seen |= bool(np.any(got != 0))
    assert seen
    g.close()
