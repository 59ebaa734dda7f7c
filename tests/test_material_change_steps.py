"""A material change inside the CPML in mid-run takes one step of its half through
the complete state; the run then goes on as before the change.  The general kernel
injects sources itself, the reduced-state one leaves them to a launch of their own,
which the launch counts show.  The fields are those of the register-pipelined kernel,
which always keeps the complete state (same recurrences up to rounding)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = {"f32": 2e-4, "f64": 1e-10}
N = (70, 22, 18)


@pytest.mark.parametrize("dtype", ["f32", "f64"])
@pytest.mark.parametrize("kinds", [(0,), (1,), (0, 1)])
def test_one_step_on_the_complete_state(kh, gpu_lib, monkeypatch, dtype, kinds):
    from khronos_gb300.device import GpuSim

    srcs = [kh.UniformSource(time_profile=kh.GaussianPulseSource(fcen=0.8, fwidth=0.2), component=c,
                             center=(0.1, 0.05, 0), size=(0, 1.0, 0.6)) for c in (kh.EY, kh.HX)]
    sp = kh.Simulation(cell_size=tuple(a / 10 for a in N), resolution=10, sources=srcs,
                       boundaries=[[0.5, 0.5], [0.4, 0.4], [0.3, 0.5]], dtype=dtype).spec()
    assert tuple(sp.n) == N
    rng = np.random.default_rng(7)
    for kind in (0, 1):
        for c in range(3):  # values exact in single precision
            sp.materials.append((kind, c, rng.integers(16, 32, size=N) / 32.0))
    a = GpuSim(sp, lib=gpu_lib)
    monkeypatch.setenv("KHRONOS_GB300_KERNEL", "simt")
    b = GpuSim(sp, lib=gpu_lib)

    def launches(g, n):
        before = g.launches
        g.step(n)
        return g.launches - before

    for g in (a, b):
        g.step(40)
    assert launches(a, 1) == 4  # two halves, two source launches
    b.step(1)
    for value in (0.25, 0.75):
        for g in (a, b):
            for kind in kinds:
                for c in range(3):
                    g.update_material_box(kind, c, (0, 0, 0), np.full((N[0], 9, N[2]), value))
        assert launches(a, 1) == 4 - len(kinds)
        assert launches(a, 7) == 28
        b.step(8)
    assert a.sources_active
    fa, fb = [a.field(c) for c in range(6)], [b.field(c) for c in range(6)]
    for grp in ((0, 1, 2), (3, 4, 5)):
        scale = np.sqrt(sum(np.sum(fb[c] ** 2) for c in grp))
        assert scale > 0
        for c in grp:
            assert np.linalg.norm(fa[c] - fb[c]) <= TOL[dtype] * scale, c
    a.close()
    b.close()
