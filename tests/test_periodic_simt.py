"""The register-pipelined kernel (KHRONOS_GB300_KERNEL=simt) on periodic axes against the
oracle: the last pair of a row takes its x neighbour from the ghost layer also where it is
not a warp's last lane (nx even, no multiple of 64)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = {"f32": 2e-4, "f64": 1e-10}


@pytest.mark.parametrize("dtype", ["f32", "f64"])
@pytest.mark.parametrize("mask", [1, 3, 7])
@pytest.mark.parametrize("n", [(6, 5, 70), (64, 8, 12), (65, 13, 9), (66, 7, 9), (128, 3, 5), (1, 9, 8)])
def test_same_as_the_oracle(kh, oracle, gpu_lib, monkeypatch, dtype, mask, n):
    from khronos_gb300.device import GpuSim

    per = [bool(mask >> a & 1) for a in range(3)]
    bnd = [[0.2, 0.2] if not per[a] and n[a] > 6 else [0.0, 0.0] for a in range(3)]
    srcs = [kh.UniformSource(time_profile=kh.GaussianPulseSource(fcen=0.8, fwidth=0.6), component=c,
                             center=(0, 0, 0), size=s)
            for c, s in ((kh.EX, (n[0] / 10, n[1] / 10, 0)), (kh.EY, (0, n[1] / 10, n[2] / 10)), (kh.HZ, (0.1, 0, 0)))]
    sp = kh.Simulation(cell_size=tuple(a / 10 for a in n), resolution=10, sources=srcs, boundaries=bnd,
                       dtype=dtype).spec()
    assert tuple(sp.n) == n
    sp.periodic = mask
    rng = np.random.default_rng(4)
    for c in range(3):
        sp.materials.append((0, c, rng.integers(8, 32, size=n) / 32.0))
    monkeypatch.setenv("KHRONOS_GB300_KERNEL", "simt")
    a = GpuSim(sp, lib=gpu_lib)
    b = oracle.OracleSim(sp)
    for steps in (1, 34):
        a.step(steps)
        b.step(steps)
        a.synchronize()
        for grp in ((0, 1, 2), (3, 4, 5)):
            scale = np.sqrt(sum(np.sum(b.field(c) ** 2) for c in grp))
            for c in grp:
                assert np.linalg.norm(a.field(c) - b.field(c)) <= TOL[dtype] * scale, (steps, c)
    a.close()
    b.close()
