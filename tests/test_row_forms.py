"""The forms of the reduced-state row update (csrc/kh_lean.cuh) give the same bits:
a uniform material takes the straight-line rows in FP32, the same value as a per-voxel
array the branching ones.  Grids whose tiles touch the x absorber with plain columns
beside it, alone and where it meets the others."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,pml", [((60, 20, 18), (6, 0, 0)), ((60, 20, 18), (6, 5, 0)), ((60, 20, 18), (6, 0, 4)),
                                   ((131, 21, 17), (6, 5, 4)), ((131, 21, 17), (0, 5, 4))])
def test_uniform_and_per_voxel_materials(kh, gpu_lib, n, pml):
    from khronos_gb300.device import GpuSim

    src = kh.UniformSource(time_profile=kh.GaussianPulseSource(fcen=0.8, fwidth=0.6), component=kh.EZ,
                           center=(0, 0, 0), size=(0, 0, 0))
    fields = []
    for voxel in (False, True):
        sp = kh.Simulation(cell_size=tuple(a / 10 for a in n), resolution=10, sources=[src],
                           boundaries=[[w / 10, w / 10] for w in pml], dtype="f32").spec()
        assert tuple(sp.n) == n
        sp.eps_inv, sp.mu_inv = 0.6875, 0.8125
        if voxel:
            for c in range(3):
                sp.materials.append((0, c, np.full(n, 0.6875)))
                sp.materials.append((1, c, np.full(n, 0.8125)))
        g = GpuSim(sp, lib=gpu_lib)
        g.step(150)
        fields.append([g.field(c) for c in range(6)])
        g.close()
    for c in range(6):
        assert np.any(fields[0][c] != 0)
        assert np.array_equal(fields[0][c], fields[1][c]), c
