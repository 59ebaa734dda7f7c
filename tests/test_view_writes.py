"""Writes through field views: what the header says of them.  They change the simulation;
values at cells that keep B/D state are recomputed from that state at the next step.
In the absorber the reduced state keeps no D where E stands for it, so the first step of
a call has to tell a written value from the state.  Against the register-pipelined kernel, which
keeps the complete state (same recurrences up to rounding)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = {"f32": 2e-4, "f64": 1e-10}


def _spec(kh, dtype, n, pml, voxel=True, sources=True):
    srcs = [kh.UniformSource(time_profile=kh.GaussianPulseSource(fcen=0.8, fwidth=0.6), component=c,
                             center=(0.1, 0.05, 0), size=(0, 0.9 * n[1] / 10, 0.6)) for c in (kh.EY, kh.HX)]
    sp = kh.Simulation(cell_size=tuple(a / 10 for a in n), resolution=10, sources=srcs if sources else [],
                       boundaries=[[w / 10, w / 10] for w in pml], dtype=dtype).spec()
    assert tuple(sp.n) == n
    rng = np.random.default_rng(3)
    if voxel:
        for kind in (0, 1):
            for c in range(3):  # values exact in single precision
                sp.materials.append((kind, c, rng.integers(16, 32, size=n) / 32.0))
    return sp


def _same(a, b, tol):
    fa, fb = [a.field(c) for c in range(6)], [b.field(c) for c in range(6)]
    for grp in ((0, 1, 2), (3, 4, 5)):
        scale = np.sqrt(sum(np.sum(fb[c] ** 2) for c in grp))
        assert scale > 0
        for c in grp:
            assert np.linalg.norm(fa[c] - fb[c]) <= tol * scale, c


def _write(g, seed, n, scale):
    import torch

    rng = np.random.default_rng(seed)
    g.synchronize()
    for c in range(6):
        v = g.field_view(c)
        add = torch.as_tensor(rng.integers(-32, 32, size=n) / 32.0 * scale, device=v.device, dtype=v.dtype)
        v[:n[0], :n[1], :n[2]].mul_(0.5).add_(add)  # the cells that are updated, not the wall layer
    torch.cuda.synchronize()


@pytest.mark.parametrize("dtype", ["f32", "f64"])
@pytest.mark.parametrize("n,pml,voxel", [((70, 22, 18), (5, 4, 3), True), ((70, 22, 18), (5, 4, 3), False),
                                         ((61, 9, 14), (6, 0, 0), True), ((40, 14, 20), (0, 4, 5), False),
                                         ((200, 100, 60), (5, 4, 3), True)])  # more than one round of CTAs
def test_writes_in_mid_run(kh, gpu_lib, monkeypatch, dtype, n, pml, voxel):
    from khronos_gb300.device import GpuSim

    sp = _spec(kh, dtype, n, pml, voxel)
    a = GpuSim(sp, lib=gpu_lib)
    monkeypatch.setenv("KHRONOS_GB300_KERNEL", "simt")
    b = GpuSim(sp, lib=gpu_lib)
    for g in (a, b):
        g.step(25)
        _write(g, 1, n, 2.0 ** -6)
        g.step(1)
        _write(g, 2, n, 2.0 ** -6)
        g.step(9)
    _same(a, b, TOL[dtype])
    for g in (a, b):  # a written state exported, and gone on from as it is
        _write(g, 3, n, 2.0 ** -6)
        g.export_state()
        g.step(7)
        if voxel:
            _write(g, 4, n, 2.0 ** -6)
            g.update_material_box(0, 1, (0, 0, 0), np.full((n[0], 3, n[2]), 0.75))
        g.step(1)
        _write(g, 5, n, 2.0 ** -6)
        g.step(4)
        g.step_timed(6)
    _same(a, b, TOL[dtype])
    a.close()
    b.close()


@pytest.mark.parametrize("dtype", ["f32", "f64"])
@pytest.mark.parametrize("gap", [False, True])
def test_initial_fields(kh, gpu_lib, monkeypatch, dtype, gap):
    from khronos_gb300.device import GpuSim

    n = (70, 22, 18)
    sp = _spec(kh, dtype, n, (5, 4, 3), sources=False)
    if gap:  # an undamped layer between damped ones
        for sg in (sp.sigma_b, sp.sigma_d):
            for a in range(3):
                sg[a] = np.array(sg[a])
                sg[a][1] = sg[a][n[a] - 2] = 0.0
    a = GpuSim(sp, lib=gpu_lib)
    monkeypatch.setenv("KHRONOS_GB300_KERNEL", "simt")
    b = GpuSim(sp, lib=gpu_lib)
    for g in (a, b):
        _write(g, 1, n, 1.0)
        g.step(30)
    _same(a, b, TOL[dtype])
    for g in (a, b):
        g.reset()
        _write(g, 2, n, 1.0)
        g.step(12)
    _same(a, b, TOL[dtype])
    a.close()
    b.close()


@pytest.mark.parametrize("dtype", ["f32", "f64"])
@pytest.mark.parametrize("periodic", [0, 6])
def test_views_that_are_only_read_change_no_bits(kh, gpu_lib, dtype, periodic):
    from khronos_gb300.device import GpuSim

    n = (70, 22, 18)
    sp = _spec(kh, dtype, n, (5, 0, 0) if periodic else (5, 4, 3))
    sp.periodic = periodic
    a, b = GpuSim(sp, lib=gpu_lib), GpuSim(sp, lib=gpu_lib)
    views = [a.field_view(c) for c in range(6)]
    for steps in (1, 30, 2, 1, 150):
        a.step(steps)
        b.step(steps)
        a.synchronize()
        for c in range(6):
            assert np.array_equal(a.field(c), b.field(c)), (steps, c)
            assert np.array_equal(views[c].double().cpu().numpy(), a.field(c))
    del views
    a.close()
    b.close()


@pytest.mark.parametrize("n", [(61, 9, 14), (130, 15, 6)])
def test_wall_layers_of_a_closed_box(kh, gpu_lib, monkeypatch, n):
    """Values written into the staggered wall layers (and the ring below) act on every
    step, whole steps through the second set of arrays as half-steps: the same bits."""
    import torch

    from khronos_gb300.device import GpuSim

    sp = _spec(kh, "f32", n, (0, 0, 0))
    sp.materials = [m for m in sp.materials if m[0] == 0]
    sp.sources = [s for s in sp.sources if s.component < 3]
    a = GpuSim(sp, lib=gpu_lib)
    monkeypatch.setenv("KHRONOS_GB300_FUSED", "0")
    b = GpuSim(sp, lib=gpu_lib)
    rng = np.random.default_rng(8)
    walls = [[rng.standard_normal((n[1] + 3, n[2] + 3, 2)), rng.standard_normal((n[0] + 3, n[2] + 3, 2)),
              rng.standard_normal((n[0] + 3, n[1] + 3, 2))] for _ in range(6)]
    for steps in (6, 7, 40):
        for g in (a, b):
            g.synchronize()
            for c in range(6):
                v = g.field_view(c, ghosted=True)  # layer -1 first, the staggered layer last
                for ax in range(3):
                    for side, at in enumerate((0, n[ax] + 1)):
                        if at < v.shape[ax]:
                            w = v.select(ax, at)
                            w.copy_(torch.as_tensor(walls[c][ax][:w.shape[0], :w.shape[1], side] * 0.01,
                                                    device=v.device, dtype=v.dtype))
            torch.cuda.synchronize()
            g.step(steps)
        for c in range(6):
            assert np.array_equal(a.field(c), b.field(c)), (steps, c)
    assert a.launches < b.launches  # whole steps were taken
    a.close()
    b.close()


def test_wall_layers_of_an_imported_state(kh, gpu_lib, monkeypatch):
    """The ring is part of a state: imported, it acts on every step without any view, and a
    reset clears it from every step."""
    import torch

    from khronos_gb300.device import GpuSim

    n = (61, 9, 14)
    sp = _spec(kh, "f32", n, (0, 0, 0))
    sp.materials = [m for m in sp.materials if m[0] == 0]
    sp.sources = [s for s in sp.sources if s.component < 3]
    first = GpuSim(sp, lib=gpu_lib)
    first.step(6)
    first.synchronize()
    rng = np.random.default_rng(8)
    for c in range(3):
        v = first.field_view(c)
        for ax in range(3):
            if v.shape[ax] > n[ax]:
                w = v.select(ax, n[ax])
                w.copy_(torch.as_tensor(rng.standard_normal(tuple(w.shape)), device=v.device, dtype=v.dtype))
    torch.cuda.synchronize()
    blob = first.export_state()
    first.close()
    a = GpuSim(sp, lib=gpu_lib)
    monkeypatch.setenv("KHRONOS_GB300_FUSED", "0")
    b = GpuSim(sp, lib=gpu_lib)
    for g in (a, b):
        g.import_state(blob)
        g.step(1)
        g.step(12)
    for c in range(6):
        assert np.array_equal(a.field(c), b.field(c)), c
    for g in (a, b):
        g.reset()
        g.step(12)
    for c in range(6):
        assert np.array_equal(a.field(c), b.field(c)), c
    a.close()
    b.close()


@pytest.mark.parametrize("pml", [(5, 4, 3), (0, 0, 0)])
def test_bounds(kh, gpu_lib, pml):
    """The bounds-checked build: no index out of range in the steps that mind views, the
    copies outside of steps, the import check and the ring, and the same bits."""
    import ctypes as C

    from khronos_gb300 import _abi, build
    from khronos_gb300.device import GpuSim

    checked = _abi.load(build.build(bounds=True))
    n = (71, 21, 18)
    out = []
    c, i, s = C.c_int64(), C.c_int64(), C.c_int32()
    for lib in (gpu_lib, checked):
        if lib is checked:
            assert lib.kh_debug_bounds(C.byref(c), C.byref(i), C.byref(s)) == 0
        sp = _spec(kh, "f32", n, pml)
        if pml[0] == 0:  # whole steps
            sp.materials = [m for m in sp.materials if m[0] == 0]
            sp.sources = [q for q in sp.sources if q.component < 3]
        else:
            sp.materials[0][2][:9, :3] = 0.0
        g = GpuSim(sp, lib=lib)
        g.step(9)
        _write(g, 1, n, 2.0 ** -6)
        g.step(4)
        blob = g.export_state()
        g.update_material_box(0, 1, (0, 0, 0), np.full((n[0], 3, n[2]), 0.75))
        g.step(1)
        g.import_state(blob)
        g.step(5)
        out.append([g.field(q) for q in range(6)])
        g.close()
    assert checked.kh_debug_bounds(C.byref(c), C.byref(i), C.byref(s)) == 0
    assert c.value == 0, (i.value, s.value)
    for x, y in zip(*out):
        assert np.array_equal(x, y)
