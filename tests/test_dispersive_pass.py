"""The dispersive-cell pass (disp_fix_kernel), which takes the two cells of a lane
together, against the general kernel that does χ3 and poles in its own cell update
(KHRONOS_GB300_DISP_FIX=0): odd rows whose last pair is half outside, segments with χ3
only, with poles and with both, poles absent from one cell of a pair, sources on
such cells, in and out of the CPML.  The bars are those of the step kernels."""
import numpy as np
import pytest


TOL = {"f32": 2e-4, "f64": 1e-10}


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["f32", "f64"])
@pytest.mark.parametrize("nx", [23, 64, 65])
@pytest.mark.parametrize("what", ["chi3", "pole", "both"])
def test_pass_equals_general_kernel(kh, gpu_lib, monkeypatch, dtype, nx, what):
    from khronos_gb300.device import GpuSim
    from khronos_gb300.spec import PoleSpec

    srcs = [kh.UniformSource(time_profile=kh.GaussianPulseSource(fcen=0.8, fwidth=0.4), component=c,
                             center=(0.1, 0.05, 0.0), size=s) for c, s in ((kh.EZ, (0, 0, 0)), (kh.EX, (0, 1.9, 1.5)))]
    sp = kh.Simulation(cell_size=(nx / 10, 2.1, 1.7), resolution=10, sources=srcs, boundaries=[[0.4, 0.4]] * 3,
                       dtype=dtype).spec()
    i, j, k = np.indices(sp.n)
    if what != "pole":
        sp.materials.append((4, 0, np.where((k >= 5) & (k < 11) & ((i + j) % 7 != 0), 0.25, 0.0)))
    if what != "chi3":
        for q in range(2):  # a Lorentz and a Drude pole on overlapping boxes
            gp, w = 0.05 * np.pi * sp.dt, (2 * np.pi * sp.dt) ** 2 * (1 - q)
            box = (i >= nx - 9 - 4 * q) & (abs(j - 10) < 4 + q) & (k > 3 + 2 * q) & ((i + q) % 3 != 0)
            sp.poles.append(PoleSpec(coeffs=dict(gamma1_inv=1 / (1 + gp), gamma1=1 - gp, omega0_dt_sq=w,
                                                 sigma_omega0_dt_sq=w, drude_coeff=0.1 * np.pi * sp.dt ** 2,
                                                 is_drude=q), sigma=np.where(box, 0.3 + q, 0.0)))
    a = GpuSim(sp, lib=gpu_lib)
    monkeypatch.setenv("KHRONOS_GB300_DISP_FIX", "0")
    b = GpuSim(sp, lib=gpu_lib)
    a.step(90)
    b.step(90)
    for grp in ((0, 1, 2), (3, 4, 5)):
        scale = np.sqrt(sum(np.sum(b.field(c) ** 2) for c in grp))
        for c in grp:
            assert np.linalg.norm(a.field(c) - b.field(c)) <= TOL[dtype] * scale, c
    a.close()
    b.close()
