"""Whole-step launches (kh_fused.cu) on grids without CPML: the same bits as the
half-step launches (KHRONOS_GB300_FUSED=0), which the parity tests hold against the
oracle.  Sizes around the tile (60 × 7 owned cells, 2 cells per thread), z chunks of
one plane, of 64-plane groups and of the rest, odd step counts (the last step of a
call is two half-steps), sources, χ3, poles, monitors of both halves and histories."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _spec(kh, n, what):
    from khronos_gb300.spec import HistorySpec, MonitorSpec, PoleSpec

    srcs = [kh.UniformSource(time_profile=kh.GaussianPulseSource(fcen=0.8, fwidth=0.4), component=c,
                             center=(0, 0, 0), size=s)
            for c, s in ((kh.EZ, (0, 0, 0)), (kh.EY, (0, n[1] / 10, n[2] / 20)))]
    sp = kh.Simulation(cell_size=tuple(a / 10 for a in n), resolution=10, sources=srcs, dtype="f32").spec()
    assert tuple(sp.n) == n
    rng = np.random.default_rng(2)
    if what != "uniform":
        for c in range(3):
            sp.materials.append((0, c, rng.integers(8, 32, size=n) / 32.0))
    if what == "dispersive":
        sp.materials.append((4, 0, np.where(rng.random(n) < 0.1, 0.05, 0.0)))
        gp, w = 0.05 * np.pi * sp.dt, (2 * np.pi * sp.dt) ** 2
        sp.poles.append(PoleSpec(coeffs=dict(gamma1_inv=1 / (1 + gp), gamma1=1 - gp, omega0_dt_sq=w,
                                             sigma_omega0_dt_sq=w, drude_coeff=0.0, is_drude=0),
                                 sigma=np.where(rng.random(n) < 0.05, 0.4, 0.0)))
    for comp in (kh.EX, kh.HY):
        sp.monitors.append(MonitorSpec(component=comp, start=(0, 0, 1), dims=(n[0], n[1], 2),
                                       freqs=np.array([0.7, 0.8]), decimation=3))
        sp.histories.append(HistorySpec(component=comp, start=(1, 0, 0), dims=(n[0] - 1, 2, n[2]), capacity=20))
    return sp


def _run(sp, lib, chunks):
    from khronos_gb300.device import GpuSim

    g = GpuSim(sp, lib=lib)
    out = []
    for c in chunks:
        g.step(c)
        out += [g.field(q) for q in range(6)]
    out += [g.dft(m) for m in range(len(sp.monitors))] + [g.history(h, t) for h in range(2) for t in (0, 7, 19)]
    n, g = g.launches, g.close()
    return out, n


@pytest.mark.parametrize("what", ["uniform", "voxel", "dispersive"])
@pytest.mark.parametrize("n,z", [((60, 7, 5), None), ((61, 8, 3), "1"), ((121, 15, 70), None), ((120, 14, 66), "64"),
                                 ((59, 6, 2), None), ((200, 22, 65), "5"), ((13, 29, 130), None)])
def test_same_bits_as_half_steps(kh, gpu_lib, monkeypatch, n, z, what):
    sp = _spec(kh, n, what)
    if z:
        monkeypatch.setenv("KHRONOS_GB300_ZPLANES", z)
    chunks = (2, 1, 24, 31)
    got, few = _run(sp, gpu_lib, chunks)
    monkeypatch.setenv("KHRONOS_GB300_FUSED", "0")
    want, many = _run(sp, gpu_lib, chunks)
    assert few < many  # whole steps were taken
    assert any(np.any(w != 0) for w in want[-6:])
    for a, b in zip(got, want):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("what", ["uniform", "dispersive"])
def test_bounds(kh, gpu_lib, monkeypatch, what):
    """The bounds-checked build: no index out of range, the same bits."""
    import ctypes as C

    from khronos_gb300 import _abi, build

    lib = _abi.load(build.build(bounds=True))
    c, i, s = C.c_int64(), C.c_int64(), C.c_int32()
    assert lib.kh_debug_bounds(C.byref(c), C.byref(i), C.byref(s)) == 0
    sp = _spec(kh, (131, 16, 67), what)
    a, _ = _run(sp, gpu_lib, (20, 5))
    b, _ = _run(sp, lib, (20, 5))
    assert lib.kh_debug_bounds(C.byref(c), C.byref(i), C.byref(s)) == 0
    assert c.value == 0, (i.value, s.value)
    for x, y in zip(a, b):
        assert np.array_equal(x, y)
