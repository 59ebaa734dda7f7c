"""A state goes on in a simulation whose materials are not those it was made with:
materials of CPML cells changed before the import, or another simulation's state.
The reduced CPML state derives W and O from the materials, so such a state has to
be continued from the complete one.  Compared with the register-pipelined kernel, which keeps
the complete state; both are the same recurrences up to rounding (the parity bars)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = {"f32": 2e-4, "f64": 1e-10}
N = (70, 22, 18)
MAT = {"eps": 0, "mu": 1}


def _spec(kh, dtype, seed, pml=((0.5, 0.5), (0.4, 0.4), (0.3, 0.5))):
    src = kh.UniformSource(time_profile=kh.GaussianPulseSource(fcen=0.8, fwidth=0.6), component=kh.EY,
                           center=(0.1, 0.05, 0), size=(0, 1.0, 0.6))
    sp = kh.Simulation(cell_size=tuple(a / 10 for a in N), resolution=10, sources=[src],
                       boundaries=[list(b) for b in pml], dtype=dtype).spec()
    assert tuple(sp.n) == N
    rng = np.random.default_rng(seed)
    for kind in MAT.values():
        for c in range(3):  # values exact in single precision
            sp.materials.append((kind, c, rng.integers(16, 32, size=N) / 32.0))
    return sp


def _pair(sp, lib, monkeypatch):
    from khronos_gb300.device import GpuSim

    a = GpuSim(sp, lib=lib)
    monkeypatch.setenv("KHRONOS_GB300_KERNEL", "simt")
    b = GpuSim(sp, lib=lib)
    monkeypatch.delenv("KHRONOS_GB300_KERNEL")
    return a, b


def _same(a, b, tol):
    fa, fb = [a.field(c) for c in range(6)], [b.field(c) for c in range(6)]
    for grp in ((0, 1, 2), (3, 4, 5)):
        scale = np.sqrt(sum(np.sum(fb[c] ** 2) for c in grp))
        assert scale > 0
        for c in grp:
            assert np.linalg.norm(fa[c] - fb[c]) <= tol * scale, c


@pytest.mark.parametrize("dtype", ["f32", "f64"])
@pytest.mark.parametrize("what", ["eps", "mu"])
def test_state_from_before_a_material_change(kh, gpu_lib, monkeypatch, dtype, what):
    a, b = _pair(_spec(kh, dtype, 3), gpu_lib, monkeypatch)
    for s in (a, b):
        s.step(60)
        blob = s.export_state()
        for c in range(3):
            s.update_material_box(MAT[what], c, (0, 0, 0), np.full((N[0], 9, N[2]), 0.25))
        s.step(5)
        s.import_state(blob)
        s.step(31)
    _same(a, b, TOL[dtype])
    a.close()
    b.close()


@pytest.mark.parametrize("dtype", ["f32", "f64"])
@pytest.mark.parametrize("kernel", ["tma", "simt"])
def test_state_of_another_simulation(kh, gpu_lib, monkeypatch, dtype, kernel):
    """Other materials everywhere, exported by either kernel."""
    first = _pair(_spec(kh, dtype, 3), gpu_lib, monkeypatch)[kernel == "simt"]
    first.step(60)
    blob = first.export_state()
    first.close()
    a, b = _pair(_spec(kh, dtype, 4), gpu_lib, monkeypatch)
    for s in (a, b):
        s.import_state(blob)
        s.step(31)
    _same(a, b, TOL[dtype])
    a.close()
    b.close()


def test_state_of_another_absorber(kh, gpu_lib, monkeypatch):
    """The exporter's absorber is thinner: U and T of the cells that were not in it
    are not equal where the importer takes them to be."""
    thin = _pair(_spec(kh, "f64", 3, pml=((0.5, 0.5), (0.2, 0.2), (0.3, 0.5))), gpu_lib, monkeypatch)[0]
    thin.step(60)
    blob = thin.export_state()
    thin.close()
    a, b = _pair(_spec(kh, "f64", 3), gpu_lib, monkeypatch)
    for s in (a, b):
        s.import_state(blob)
        s.step(31)
    _same(a, b, TOL["f64"])
    a.close()
    b.close()


@pytest.mark.parametrize("dtype", ["f32", "f64"])
def test_own_state_continues_with_the_same_bits(kh, gpu_lib, dtype):
    """Nothing is flagged in a state of the same simulation, also late in a run: the
    fields go on bit for bit, with the launches of an undisturbed run."""
    from khronos_gb300.device import GpuSim

    sp = _spec(kh, dtype, 5)
    a, b = GpuSim(sp, lib=gpu_lib), GpuSim(sp, lib=gpu_lib)
    for steps in (40, 700):
        a.step(steps)
        b.import_state(a.export_state())
        a.step(20)
        b.step(20)
        for c in range(6):
            assert np.array_equal(a.field(c), b.field(c)), (steps, c)
    a.close()
    b.close()
