"""The reduced-state kernel in the absorber itself: faces, edges and corners (where U
lives) each against their own norm, from random fields all over the grid, so that none
is far below another.  Against the register-pipelined kernel, which keeps the complete
state.  Both round each of about ten operations a step differently; 40 steps of them
stay below 40 · 16 · eps."""
import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = {"f32": 2.0 ** -24, "f64": 2.0 ** -53}
STEPS = 40


@pytest.mark.parametrize("dtype", ["f32", "f64"])
@pytest.mark.parametrize("voxel", [False, True])
@pytest.mark.parametrize("n", [(30, 24, 26), (67, 25, 22), (130, 23, 27)])
def test_every_part_of_the_absorber(kh, gpu_lib, monkeypatch, dtype, voxel, n):
    import torch

    from khronos_gb300.device import GpuSim

    pml = (6, 7, 8)
    sp = kh.Simulation(cell_size=tuple(a / 10 for a in n), resolution=10, sources=[],
                       boundaries=[[w / 10, w / 10] for w in pml], dtype=dtype).spec()
    assert tuple(sp.n) == n
    if voxel:
        rng = np.random.default_rng(5)
        for kind in (0, 1):
            for c in range(3):  # values exact in single precision
                sp.materials.append((kind, c, rng.integers(16, 32, size=n) / 32.0))
    fields = []
    for kernel in ("tma", "simt"):
        monkeypatch.setenv("KHRONOS_GB300_KERNEL", kernel)
        g = GpuSim(sp, lib=gpu_lib)
        rng = np.random.default_rng(6)
        for c in range(6):
            v = g.field_view(c)
            v[:n[0], :n[1], :n[2]].copy_(torch.as_tensor(rng.integers(-32, 33, size=n) / 32.0, device=v.device))
        torch.cuda.synchronize()
        g.step(STEPS)
        fields.append([g.field(c)[:n[0], :n[1], :n[2]] for c in range(6)])
        g.close()
    inside = [(np.arange(n[a]) < pml[a]) | (np.arange(n[a]) >= n[a] - pml[a]) for a in range(3)]
    f = np.meshgrid(*inside, indexing="ij")
    for part in itertools.product([False, True], repeat=3):
        cells = np.logical_and.reduce([x if want else ~x for x, want in zip(f, part)])
        for grp in ((0, 1, 2), (3, 4, 5)):
            a, b = (np.array([fl[c][cells] for c in grp]) for fl in fields)
            scale = np.linalg.norm(b)
            assert scale > 0
            assert np.linalg.norm(a - b) <= STEPS * 16 * EPS[dtype] * scale, (part, grp)
