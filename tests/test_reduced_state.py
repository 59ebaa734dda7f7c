"""The reduced CPML state (csrc/kh_lean.cuh): T, U and W that follow from the
rest of the state are neither stored nor read by the step kernels.

The general kernel (KHRONOS_GB300_KERNEL=simt) keeps the complete state, so both
are run on the same inputs: whole runs, runs continued by the other kernel from
an exported state, and a material change inside the CPML in mid-run.  Both are
the same recurrences up to rounding: the parity bars of the step kernels apply
(1e-10 in FP64, 2e-4 in FP32)."""
import itertools

import numpy as np
import pytest

from conftest import rel_l2

MAT_EPS_INV = 0

TOL = {"f32": 2e-4, "f64": 1e-10}


def full_cascade(f, s, m, K):
    """O of one component under the complete cascade; f, s: (own, next, previous)."""
    t = u = w = O = 0.0
    out = []
    for k in K:
        d = k
        if f[1] and s[1]:
            un = ((1 - s[1]) * u + k) / (1 + s[1])
            d, u = un - u, un
        t = ((1 - s[2]) * t + d) / (1 + s[2]) if f[2] and s[2] else t + d
        if f[0] and s[0]:
            wn = m * t
            O, w = O + (1 + s[0]) * wn - (1 - s[0]) * w, wn
        else:
            O = m * t
        out.append(O)
    return np.array(out)


def reduced(f, s, m, K):
    """The same from T (own-axis CPML only) and U (both other axes only)."""
    a, b = [(1 - x) / (1 + x) if g else 1.0 for g, x in zip(f, s)], [1 / (1 + x) if g else 1.0 for g, x in zip(f, s)]
    t = u = O = 0.0
    out = []
    for k in K:
        d = k
        if f[1] and f[2]:
            un = a[1] * u + b[1] * k
            d, u = un - u, un
        A, B = (a[2], b[2]) if f[2] else (a[1], b[1])
        if f[0]:
            tn = A * t + B * d
            O, t = O + m * ((1 + s[0]) * tn - (1 - s[0]) * t), tn
        else:
            O = A * O + m * B * d
        out.append(O)
    return np.array(out)


@pytest.mark.parametrize("f", list(itertools.product([False, True], repeat=3)))
@pytest.mark.parametrize("zero", [None, 0, 1, 2])
def test_recurrences_agree(f, zero):
    """Every combination of CPML flags, also with σ = 0 on a flagged axis; 400
    steps of rounding in FP64 stay far below 1e-12 of the largest value."""
    rng = np.random.default_rng(5)
    s = [0.0 if a == zero else x for a, x in enumerate((0.31, 0.07, 1.4))]
    K = rng.standard_normal(400)
    x, y = full_cascade(f, s, 0.37, K), reduced(f, s, 0.37, K)
    assert np.max(np.abs(x - y)) <= 1e-12 * np.max(np.abs(x))


def _spec(kh, dtype, boundaries, size, h_source=False):
    srcs = [kh.UniformSource(time_profile=kh.GaussianPulseSource(fcen=0.8, fwidth=0.4), component=c,
                             center=(0.1, 0.05, 0.0), size=sz)
            for c, sz in ((kh.EZ, (0, 0, 0)), (kh.EX, (0, size[1] * 0.9, size[2] * 0.9)))]
    if h_source:
        srcs.append(kh.UniformSource(time_profile=kh.GaussianPulseSource(fcen=0.8, fwidth=0.4), component=kh.HY,
                                     center=(-0.3, 0.0, 0.0), size=(0, size[1] * 0.9, size[2] * 0.5)))
    mon = kh.DFTMonitor(component=kh.EY, center=(0.3, 0, 0), size=(0, 0.6, 0.6), frequencies=[0.8])
    sp = kh.Simulation(cell_size=size, resolution=10, sources=srcs, monitors=[mon], boundaries=boundaries,
                       dtype=dtype).spec()
    rng = np.random.default_rng(11)
    for c in range(3):  # per-voxel ε⁻¹, values exact in single precision
        sp.materials.append((MAT_EPS_INV, c, rng.integers(8, 32, size=sp.n) / 32.0))
    return sp


def _compare(a, b, tol, ncomp=6):
    fa, fb = [a.field(c) for c in range(ncomp)], [b.field(c) for c in range(ncomp)]
    for grp in ((0, 1, 2), (3, 4, 5)):
        scale = np.sqrt(sum(np.sum(fb[c] ** 2) for c in grp))
        for c in grp:  # H is exactly zero in both after the first step without an H source
            assert np.linalg.norm(fa[c] - fb[c]) <= tol * scale, c
    assert rel_l2(a.dft(0), b.dft(0)) <= tol


SHAPES = [  # cell size (10 cells per unit) and CPML widths: edges of the 64 × 4 tiles, remainders, single sides
    ((6.5, 2.1, 1.7), ((0.5, 0.5), (0.5, 0.5), (0.5, 0.5))),
    ((3.3, 1.9, 6.6), ((0.3, 0.0), (0.0, 0.7), (0.4, 0.4))),
    ((12.9, 1.3, 1.5), ((0.6, 0.6), (0.0, 0.0), (0.2, 0.0))),
    ((1.9, 1.7, 1.3), ((0.0, 0.0), (0.5, 0.5), (0.0, 0.0))),
]


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["f32", "f64"])
@pytest.mark.parametrize("shape", range(len(SHAPES)))
def test_same_run_as_the_general_kernel(kh, gpu_lib, monkeypatch, dtype, shape):
    from khronos_gb300.device import GpuSim

    size, bnd = SHAPES[shape]
    sp = _spec(kh, dtype, [list(b) for b in bnd], size, h_source=shape % 2 == 0)
    a = GpuSim(sp, lib=gpu_lib)
    monkeypatch.setenv("KHRONOS_GB300_KERNEL", "simt")
    b = GpuSim(sp, lib=gpu_lib)
    for n in (1, 50, 69):
        a.step(n)
        b.step(n)
        _compare(a, b, TOL[dtype])
    a.close()
    b.close()


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["f32", "f64"])
def test_state_passes_between_the_kernels(kh, gpu_lib, monkeypatch, dtype):
    """A state exported by either kernel is continued by the other, the size of
    the exported state is the same, and exporting disturbs nothing."""
    from khronos_gb300.device import GpuSim

    size, bnd = SHAPES[0]
    sp = _spec(kh, dtype, [list(b) for b in bnd], size)
    red = [GpuSim(sp, lib=gpu_lib) for _ in range(2)]
    monkeypatch.setenv("KHRONOS_GB300_KERNEL", "simt")
    gen = [GpuSim(sp, lib=gpu_lib) for _ in range(2)]
    red[0].step(45)
    gen[0].step(45)
    blob_r, blob_g = red[0].export_state(), gen[0].export_state()
    assert len(blob_r) == len(blob_g)
    red[1].import_state(blob_g)
    gen[1].import_state(blob_r)
    for s in red + gen:
        s.step(60)
    for s in (red[0], red[1], gen[1]):
        _compare(s, gen[0], TOL[dtype])
    for s in red + gen:
        s.close()


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["f32", "f64"])
def test_material_change_inside_the_cpml(kh, gpu_lib, monkeypatch, dtype):
    """ε⁻¹ changed in mid-run on cells of the CPML: the same as on the complete
    state, also after an export, and a reset goes back to the reduced state."""
    from khronos_gb300.device import GpuSim

    size, bnd = SHAPES[0]
    sp = _spec(kh, dtype, [list(b) for b in bnd], size)
    a, c = GpuSim(sp, lib=gpu_lib), GpuSim(sp, lib=gpu_lib)
    monkeypatch.setenv("KHRONOS_GB300_KERNEL", "simt")
    b = GpuSim(sp, lib=gpu_lib)
    start, dims = (0, 0, 0), (sp.n[0], 9, 9)
    for s in (a, b):
        s.step(40)
        for comp in range(3):
            s.update_material_box(MAT_EPS_INV, comp, start, np.full(dims, 0.6))
        s.step(20)
    c.import_state(a.export_state())
    for comp in range(3):
        c.update_material_box(MAT_EPS_INV, comp, start, np.full(dims, 0.6))
    for s in (a, b, c):
        s.step(35)
    _compare(a, b, TOL[dtype])
    _compare(c, b, TOL[dtype])
    for s in (a, b):
        s.reset()
        s.step(50)
    _compare(a, b, TOL[dtype])
    for s in (a, b, c):
        s.close()
