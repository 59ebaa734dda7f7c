"""ε⁻¹ or μ⁻¹ = 0 on cells of the absorber (a perfect conductor): their fields stay zero,
but D and B go on, and count again when the material changes in mid-run.  Against the
register-pipelined kernel, which keeps the complete state (the parity bars)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = {"f32": 2e-4, "f64": 1e-10}
N = (70, 22, 18)


@pytest.mark.parametrize("dtype", ["f32", "f64"])
@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("sources", [True, False])
@pytest.mark.parametrize("views", [True, False])
def test_zero_material_in_the_absorber(kh, gpu_lib, monkeypatch, dtype, kind, sources, views):
    import torch

    from khronos_gb300.device import GpuSim

    src = kh.UniformSource(time_profile=kh.GaussianPulseSource(fcen=0.8, fwidth=0.6), component=kh.EY,
                           center=(0.1, 0.05, 0), size=(0, 1.0, 0.6))
    sp = kh.Simulation(cell_size=tuple(a / 10 for a in N), resolution=10, sources=[src] if sources else [],
                       boundaries=[[0.5, 0.5], [0.4, 0.4], [0.3, 0.5]], dtype=dtype).spec()
    assert tuple(sp.n) == N
    rng = np.random.default_rng(9)
    for k in (0, 1):
        for c in range(3):  # values exact in single precision
            m = rng.integers(16, 32, size=N) / 32.0
            if k == kind:
                m[20:40, :6, :] = 0.0
            sp.materials.append((k, c, m))
    start = [rng.integers(-32, 33, size=N) / 32.0 for _ in range(6)]
    box = {"dead": (20, 0, 0), "live": (45, 0, 0)}
    out = []
    for kernel in ("tma", "simt"):
        monkeypatch.setenv("KHRONOS_GB300_KERNEL", kernel)
        g = GpuSim(sp, lib=gpu_lib)
        if not sources:  # something has to be in the grid
            for c in range(6):
                v = g.field_view(c)
                v[:N[0], :N[1], :N[2]].copy_(torch.as_tensor(start[c], device=v.device))
            torch.cuda.synchronize()
        elif views:
            g.field_view(0)
        g.step(40)
        for c in range(3):
            g.update_material_box(kind, c, box["dead"], np.full((15, 6, N[2]), 0.5))
            g.update_material_box(kind, c, box["live"], np.zeros((10, 6, N[2])))
        g.step(1)
        g.step(19)
        for c in range(3):
            g.update_material_box(kind, c, box["live"], np.full((10, 6, N[2]), 0.75))
        g.step(15)
        out.append([g.field(c) for c in range(6)])
        g.close()
    for grp in ((0, 1, 2), (3, 4, 5)):
        scale = np.sqrt(sum(np.sum(out[1][c] ** 2) for c in grp))
        assert scale > 0
        for c in grp:
            assert np.linalg.norm(out[0][c] - out[1][c]) <= TOL[dtype] * scale, c
