"""Periodic ghost layers written by the half-step that updates the faces (and again by
the source kernel for source cells on them), against the oracle's wrap: every mask of axes, one-cell and odd extents, tiles that end on
and past a face, a source plane over whole faces and in the absorber of the other axis.
The layers themselves are copies: bit equality with the face across."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = {"f32": 2e-4, "f64": 1e-10}


@pytest.mark.parametrize("dtype", ["f32", "f64"])
@pytest.mark.parametrize("mask", range(1, 8))
@pytest.mark.parametrize("n", [(64, 8, 12), (65, 13, 9), (3, 30, 7), (131, 1, 10), (6, 5, 70)])
def test_same_as_the_oracle(kh, oracle, gpu_lib, dtype, mask, n):
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
    for c in range(6):
        # ghosted view: index 0 is layer -1; the reference wraps the centre range only
        v = a.field_view(c, ghosted=True).double().cpu().numpy()
        core = v[1:n[0] + 1, 1:n[1] + 1, 1:n[2] + 1]
        for ax in range(3):
            sl = [slice(1, m + 1) for m in n]
            sl[ax] = 0
            want = np.take(core, -1, axis=ax) if per[ax] else 0.0 * np.take(core, -1, axis=ax)
            assert np.array_equal(v[tuple(sl)], want), (c, ax)
    a.close()
    b.close()
