"""Words a cell and step of the traffic model on closed boxes: 12 where whole steps are
taken, 18 in half-steps (3 more with per-voxel ε); the split is that of half-steps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,fused,words", [("f32", "1", 12), ("f32", "0", 18), ("f64", "1", 18)])
@pytest.mark.parametrize("voxel", [0, 3])
def test_closed_box(kh, gpu_lib, monkeypatch, dtype, fused, words, voxel):
    from khronos_gb300.device import GpuSim

    monkeypatch.setenv("KHRONOS_GB300_FUSED", fused)
    sp = kh.Simulation(cell_size=(3.3, 2.1, 1.7), resolution=10, sources=[], dtype=dtype).spec()
    if voxel:
        for c in range(3):
            sp.materials.append((0, c, np.full(sp.n, 0.5)))
    g = GpuSim(sp, lib=gpu_lib)
    word = np.prod(sp.n) * (4 if dtype == "f32" else 8)
    assert g.model_bytes_per_step() == (words + voxel) * word
    assert sum(g.model_bytes_split()) == (18 + voxel) * word
    g.close()
