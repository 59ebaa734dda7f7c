"""One H half-step of the reduced-state kernel against its formula, in FP32, bit by bit: a
damped component is fma(A, O, m·(B·K)), rounded once at the size of O, a plain one
fma(m, K, O).  The multiply-adds are evaluated in double precision, where their products
are exact, and rounded to single; the rounding of the double sum first can change one
result in about 2^29."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

F, D = np.float32, np.float64


def _fma(a, b, c):
    return (a.astype(D) * b.astype(D) + c.astype(D)).astype(F)


@pytest.mark.parametrize("voxel", [False, True])
@pytest.mark.parametrize("axis,n", [(0, (70, 20, 18)), (1, (70, 26, 18)), (2, (70, 20, 26))])
def test_rounding_of_a_half_step(kh, gpu_lib, axis, n, voxel):
    from khronos_gb300.device import GpuSim

    src = kh.UniformSource(time_profile=kh.GaussianPulseSource(fcen=0.8, fwidth=0.6), component=kh.EZ,
                           center=(0, 0, 0), size=(0, 0, 0))
    bounds = [[0.6, 0.6] if a == axis else [0.0, 0.0] for a in range(3)]
    sp = kh.Simulation(cell_size=tuple(a / 10 for a in n), resolution=10, sources=[src], boundaries=bounds,
                       dtype="f32").spec()
    assert tuple(sp.n) == n
    rng = np.random.default_rng(5)
    sp.mu_inv = 0.8125
    mu = [np.full(n, F(0.8125)) for _ in range(3)]
    if voxel:
        mu = [(rng.integers(16, 32, size=n) / 32.0).astype(F) for _ in range(3)]
        for c in range(3):
            sp.materials.append((1, c, mu[c].astype(D)))
    g = GpuSim(sp, lib=gpu_lib)

    def cells(c):  # without the wall layers
        return g.field(c)[:n[0], :n[1], :n[2]].astype(F)

    g.step(120)
    f = [cells(c) for c in range(6)]
    g.step(1)
    got = [cells(c) for c in range(3, 6)]
    g.close()
    cd = [F(sp.dt) * (F(1) / F(d)) for d in sp.delta]
    K = []
    for c in range(3):  # cd_b (A_a(+b) - A_a) - cd_a (A_b(+a) - A_b), away from the high walls
        a, b = (c + 1) % 3, (c + 2) % 3
        da = np.diff(f[a], axis=b, append=F(0))
        db = np.diff(f[b], axis=a, append=F(0))
        K.append(_fma(np.full(n, cd[b]), da, -(cd[a] * db)))
    s = np.asarray(sp.sigma_b[axis], dtype=F)
    assert np.count_nonzero(s) >= 8
    shape = [1, 1, 1]
    shape[axis] = n[axis]
    s = np.broadcast_to(s.reshape(shape), n)
    B = F(1) / (F(1) + s)
    A = (F(1) - s) * B
    inner = (slice(0, -1),) * 3
    for c in range(3):
        if c == axis:  # goes through T in the absorber
            continue
        O = f[3 + c]
        want = np.where(s != 0, _fma(A, O, mu[c] * (B * K[c])), _fma(mu[c], K[c], O))[inner]
        assert np.count_nonzero(want[(s != 0)[inner]]) > 1000
        assert np.count_nonzero(want != got[c][inner]) <= 1, c
