"""Performance cases of the FDTD step loop and what surrounds it.

Every case is a piece of work a user has the framework do through its public
entry points (``device.GpuSim``, ``serve.run_batch_concurrent``):

* ``solve``    one simulation that a program keeps and runs again for new
               excitations or as one point of a sweep: ``reset``, N steps, the
               flux spectra, the six fields in place on the device;
* ``watch``    a run stepped one step at a time, with the monitors' norms read
               whenever they were updated (how a decay criterion drives a run);
* ``new``      a one-off run from host arrays: create, prepare, N steps, the
               fields and DFT arrays copied to the host, release;
* ``gradient`` a windowed adjoint gradient: forward run with recorded design
               voxels, adjoint run from the objective cells, correlation;
* ``serve``    a batch of independent requests through the request server.

Sizes are those of ``configs.py`` (64³ dipole, 320×192×128 waveguide, 256³
dispersive, 256×256×128 periodic slab, the serving grids, the bend), of the FP64
parity runs, a ragged grid as in the tests, a closed cavity and one grid well
above the last-level cache.  Materials are random spheres over a background (as
in the serving stream), sources are tilted dipoles or current planes with a
Gaussian pulse that is switched off inside the run, monitors are flux planes.

Values that an FP32 run hands back in FP64 arrays (fluxes, DFT arrays, norms,
host copies of fields) are returned in single precision, which is what they
hold.
"""
import math
import random  # noqa: F401  (the type of draw()'s argument)

import numpy as np
import torch

RES = 16            # cells per µm: Δ = 1/16 and Δt = 1/32 are exact in FP32
DELTA = 1.0 / RES
DT = 0.5 * DELTA
FCEN = 0.5


def _package():
    import __graft_entry__

    return __graft_entry__.package()


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


# --------------------------------------------------------------------------
# cases

def _case(kind, n, steps, **kw):
    c = dict(kind=kind, nx=n[0], ny=n[1], nz=n[2], steps=steps, dtype="f32", pml=12, voxel=True, mu=False,
             chi3=False, poles=0, periodic=0, source="plane", h_source=False, nf=21)
    c.update(kw)
    return c


def listed():
    return [
        # the smallest run of the configurations and of the serving stream: launches and latency count
        dict(name="dipole_64", **_case("solve", (64, 64, 64), 256, pml=10, voxel=False, source="dipole", nf=3)),
        # the headline workload: per-voxel ε, a current plane, two flux planes at 21 frequencies
        dict(name="waveguide_320x192x128", **_case("solve", (320, 192, 128), 96)),
        # Kerr slab through the whole cross-section, Lorentz and Drude spheres
        dict(name="dispersive_256", **_case("solve", (256, 256, 256), 40, chi3=True, poles=2, nf=11)),
        # supercell wrapped along x and y, absorber along z only
        dict(name="periodic_256x256x128", **_case("solve", (256, 256, 128), 64, periodic=3)),
        # odd extents, asymmetric absorber, per-voxel μ, electric and magnetic currents
        dict(name="ragged_181x97x75", **_case("solve", (181, 97, 75), 120, pml=9, mu=True, h_source=True, nf=5)),
        # closed metallic box, uniform medium, no absorber: the plain update alone
        dict(name="cavity_216x200x168", **_case("solve", (216, 200, 168), 100, pml=0, voxel=False, source="dipole",
                                                nf=5)),
        # a device-scale run far above the caches
        dict(name="large_512x384x256", **_case("solve", (512, 384, 256), 24)),
        # the double-precision run that single-precision results are held against
        dict(name="waveguide_f64_240x144x96", **_case("solve", (240, 144, 96), 32, dtype="f64", nf=5)),
        # a run under a decay criterion: one step per call, norms after every monitor update
        dict(name="watch_96", **_case("watch", (96, 96, 96), 64, pml=10, source="dipole", nf=5)),
        # one-off run from host arrays, everything read back
        dict(name="new_160x160x96", **_case("new", (160, 160, 96), 64, pml=10, nf=5)),
        # inverse design: gradient of an objective with respect to every design voxel
        dict(name="gradient_200x200x64", **_case("gradient", (200, 200, 64), 128)),
        # the serving stream's grids, two requests each
        dict(name="serve_10", **_case("serve", (160, 160, 96), 160, pml=10, source="dipole", nf=5, requests=10)),
    ]


def draw(rng):
    def size(lo, hi, most=30_000_000):
        while True:
            n = tuple(int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))) for _ in range(3))
            if n[0] * n[1] * n[2] <= most:
                return n

    kind = rng.choice(["solve"] * 7 + ["watch", "new", "gradient", "serve"])
    if kind == "serve":
        return _case("serve", (160, 160, 96), rng.randrange(64, 160), pml=10, source="dipole", nf=rng.randrange(3, 8),
                     requests=rng.randrange(4, 10))
    if kind == "watch":
        return _case("watch", size(48, 160, 3_000_000), rng.randrange(24, 64), pml=10, source="dipole",
                     nf=rng.randrange(2, 8))
    if kind == "new":
        return _case("new", size(64, 200, 4_000_000), rng.randrange(16, 96), pml=10, nf=rng.randrange(2, 8))
    if kind == "gradient":
        return _case("gradient", size(64, 200, 3_000_000), rng.randrange(64, 128))
    dtype = "f64" if rng.random() < 0.15 else "f32"
    n = size(48, 420, 6_000_000 if dtype == "f64" else 30_000_000)
    # runs from 16 to 256 steps, the longer ones on the smaller grids
    steps = max(16, min(rng.randrange(48, 257), int((1.1e8 if dtype == "f64" else 1.1e9) / (n[0] * n[1] * n[2]))))
    what = rng.choice(["waveguide"] * 3 + ["dispersive", "periodic", "magnetic", "cavity"])
    c = _case("solve", n, steps, dtype=dtype, pml=rng.randrange(8, 14), nf=rng.randrange(1, 22),
              source=rng.choice(["dipole", "plane"]), voxel=rng.random() < 0.8)
    if what == "dispersive":
        c.update(chi3=rng.random() < 0.7, poles=rng.randrange(0, 3), voxel=True)
    elif what == "periodic":
        c.update(periodic=rng.choice([1, 2, 3, 4, 6]), source="plane")
    elif what == "magnetic":
        c.update(mu=rng.random() < 0.5, h_source=True)
    elif what == "cavity":
        c.update(pml=0)
    return c


# --------------------------------------------------------------------------
# inputs, from the case and the seed alone

SERVING_GRIDS = [(64, 64, 64), (96, 96, 96), (128, 128, 128), (160, 160, 96), (256, 128, 64)]
COMP_OFF = [(0.5, 0, 0), (0, 0.5, 0), (0, 0, 0.5)]  # Yee positions of Ex, Ey, Ez in cells


def _np_dtype(case):
    return np.float32 if case["dtype"] == "f32" else np.float64


def _widths(case):
    """Absorber cells on the low and the high side of each axis."""
    lo, hi = [], []
    for a in range(3):
        w = 0 if (case["periodic"] >> a) & 1 else case["pml"]
        lo.append(w)
        hi.append(max(0, w - 2) if case["h_source"] and a == 1 else w)  # asymmetric along y on the ragged grid
    return lo, hi


def _sigma(n, lo, hi, T):
    """Quadratic absorber profile (already scaled by Δt/2), positive on every absorber cell."""
    s = np.zeros(n)
    smax = 0.8 * 3 / DELTA * DT / 2
    for i in range(lo):
        s[i] = smax * ((lo - i) / lo) ** 2
    for i in range(hi):
        s[n - 1 - i] = smax * ((hi - i) / hi) ** 2
    return s.astype(T).astype(np.float64)


def _spheres(n, rng, count, rmax=None):
    out = []
    m = min(n)
    for _ in range(count):
        r = float(rng.uniform(0.06, 0.2)) * m if rmax is None else float(rng.uniform(0.4, 1.0)) * rmax
        out.append(([float(rng.uniform(0.2, 0.8)) * n[a] for a in range(3)], r, float(rng.uniform(2, 12))))
    return out


def _paint(n, base, spheres, off, values=None):
    """(nz, ny, nx) array: `base` with the spheres painted over it (first one wins)."""
    dev = _dev()
    g = [torch.arange(n[a], device=dev, dtype=torch.float32) + float(off[a]) for a in range(3)]
    out = torch.full((n[2], n[1], n[0]), float(base), device=dev, dtype=torch.float64)
    for q in reversed(range(len(spheres))):
        c, r, e = spheres[q]
        d2 = ((g[0] - c[0]) ** 2)[None, None, :] + ((g[1] - c[1]) ** 2)[None, :, None] + ((g[2] - c[2]) ** 2)[:, None, None]
        out[d2 <= r * r] = e if values is None else values[q]
    return out


def _inputs(case, seed):
    """Everything one simulation is made of, arrays as torch (nz, ny, nx) FP64
    tensors that hold values of the run's precision."""
    rng = np.random.default_rng(int(seed))
    n = (case["nx"], case["ny"], case["nz"])
    T = _np_dtype(case)
    tt = torch.float32 if T is np.float32 else torch.float64

    def rounded(a):
        return a.to(tt).to(torch.float64)

    lo, hi = _widths(case)
    s = dict(n=n, lo=lo, hi=hi, sigma=[_sigma(n[a], lo[a], hi[a], T) for a in range(3)], eps=None, mu=None,
             chi3=None, poles=[], sources=[], monitors=[], planes=[], histories=[],
             eps_inv=float(T(1.0 / 2.25)) if not case["voxel"] else 1.0)
    spheres = _spheres(n, rng, int(rng.integers(4, 13)))
    if case["voxel"]:
        s["eps"] = [rounded(1.0 / _paint(n, 2.085, spheres, COMP_OFF[c])) for c in range(3)]
    if case["mu"]:
        magnets = _spheres(n, rng, 3)
        s["mu"] = [rounded(1.0 / _paint(n, 1.0, magnets, COMP_OFF[(c + 1) % 3], values=[1.5, 1.2, 2.0]))
                   for c in range(3)]
    if case["chi3"]:
        third = torch.zeros((n[2], n[1], n[0]), device=_dev(), dtype=torch.float64)
        third[int(0.42 * n[2]):max(int(0.42 * n[2]) + 1, int(0.58 * n[2]))] = 1e-3
        s["chi3"] = rounded(third)
    for p in range(case["poles"]):
        m = min(n)
        inner = [([float(rng.uniform(0.35, 0.65)) * n[a] for a in range(3)], 0.12 * m, 1.0) for _ in range(4)]
        sig = _paint(n, 0.0, inner, (0, 0, 0))
        w0, gamma, strength = (1.0, 0.05, 0.6) if p == 0 else (0.0, 0.1, 30.0)
        for a in range(3):  # no poles in the absorber
            view = sig.movedim(2 - a, 0)
            view[:lo[a]] = 0.0
            if hi[a]:
                view[n[a] - hi[a]:] = 0.0
        gp = gamma * math.pi * DT
        s["poles"].append(dict(coeffs=dict(gamma1_inv=1.0 / (1.0 + gp), gamma1=1.0 - gp,
                                           omega0_dt_sq=(2 * math.pi * w0 * DT) ** 2,
                                           sigma_omega0_dt_sq=(2 * math.pi * w0 * DT) ** 2,
                                           drude_coeff=gamma * 2 * math.pi * DT * DT,
                                           is_drude=1 if w0 == 0 else 0), sigma=rounded(sig * strength)))
    # a tilted dipole, or a current plane with a Gaussian profile
    width = float(T(case["steps"] * DT / 9.0))
    pulse = dict(fcen=float(T(FCEN)), width=width, peak=float(T(5 * width)), cutoff=float(T(5 * width)))
    tilt = rng.uniform(0.5, 1.0, size=3)
    normal = 2 if case["periodic"] & 1 else 0  # the plane's normal axis
    for c in range(3):
        if case["source"] == "dipole":
            start = [int(0.4 * n[a]) + int(rng.integers(0, max(1, n[a] // 8))) for a in range(3)]
            amp = np.full((1, 1, 1), tilt[c])
        else:
            start = [lo[a] + 1 if not (case["periodic"] >> a) & 1 else 0 for a in range(3)]
            dims = [n[a] - lo[a] - hi[a] - 2 if not (case["periodic"] >> a) & 1 else n[a] for a in range(3)]
            start[normal] = int(0.35 * n[normal])
            dims[normal] = 1
            ax = [(np.arange(d) + st - 0.5 * n[a]) / (0.3 * n[a]) for a, (d, st) in enumerate(zip(dims, start))]
            ax[normal] = np.zeros(1)
            amp = tilt[c] * np.exp(-(ax[0][:, None, None] ** 2 + ax[1][None, :, None] ** 2 + ax[2][None, None, :] ** 2))
        s["sources"].append(dict(comp=c, start=start, amp=amp.astype(T).astype(np.float64), **pulse))
    if case["h_source"]:
        for q in list(s["sources"]):
            s["sources"].append(dict(q, comp=3 + q["comp"], amp=(0.5 * q["amp"][::-1, ::-1, ::-1]).astype(T).astype(np.float64)))
    # flux planes: E and H of the two tangential axes
    fmax = FCEN * 1.25
    freqs = np.linspace(0.75 * FCEN, fmax, case["nf"]) if case["nf"] > 1 else np.array([FCEN])
    freqs = freqs.astype(T).astype(np.float64)
    dec = max(1, int(1.0 / (2 * fmax * DT) / 4))
    a1, a2 = [a for a in range(3) if a != normal]
    at = s["sources"][0]["start"][normal]
    for pos in (at - 4, at + 8) if case["source"] == "plane" else (at + 5,):
        start = [lo[a] + 1 for a in range(3)]
        dims = [max(1, n[a] - lo[a] - hi[a] - 2) for a in range(3)]
        start[normal] = pos
        dims[normal] = 1
        ids = []
        for comp in (a1, a2, 3 + a1, 3 + a2):
            ids.append(len(s["monitors"]))
            s["monitors"].append(dict(comp=comp, start=list(start), dims=list(dims), freqs=freqs, dec=dec))
        s["planes"].append((ids, normal, DELTA * DELTA))
    return s


def _gradient_inputs(case, seed):
    """Forward simulation with recorded design voxels and adjoint simulation
    driven on the objective cells by a table."""
    fwd = _inputs(case, seed)
    n = fwd["n"]
    rng = np.random.default_rng(int(seed) + 7919)
    dims = [max(2, int(0.3 * n[0])), max(2, int(0.3 * n[1])), max(2, int(0.18 * n[2]))]
    start = [(n[a] - dims[a]) // 2 for a in range(3)]
    fwd["monitors"], fwd["planes"] = [], []
    fwd["histories"] = [dict(comp=c, start=start, dims=dims) for c in range(3)]
    adj = dict(fwd, sources=[])
    T = _np_dtype(case)
    odims = [max(1, n[0] // 5), 1, max(1, n[2] // 5)]
    ostart = [(n[0] - odims[0]) // 2, int(0.62 * n[1]), (n[2] - odims[2]) // 2]
    t = (np.arange(case["steps"]) + 0.5) * DT
    f = np.exp(-((t - t[-1] / 3) / (t[-1] / 6)) ** 2)
    table = np.stack([np.zeros_like(t), f * np.cos(2 * math.pi * FCEN * t)], axis=1).astype(T).astype(np.float64)
    for c in range(3):
        amp = rng.uniform(0.2, 1.0, size=odims).astype(T).astype(np.float64)
        adj["sources"].append(dict(comp=c, start=ostart, amp=amp, fcen=FCEN, width=0.0, peak=0.0,
                                   cutoff=1e6, table=table))
    return fwd, adj


def _serve_cases(case):
    out = []
    for i in range(case["requests"]):
        g = SERVING_GRIDS[i % len(SERVING_GRIDS)]
        c = dict(case, kind="solve", nx=g[0], ny=g[1], nz=g[2], steps=case["steps"] + 13 * (i % 3))
        out.append(c)
    return out


# --------------------------------------------------------------------------
# the framework's side

def _host(a, dtype):
    """(nz, ny, nx) device tensor -> host array indexed [i, j, k], x fastest."""
    return a.to(dtype).cpu().numpy().transpose(2, 1, 0)


def _spec(case, s):
    _package()
    from khronos_gb300 import spec as S

    f32 = case["dtype"] == "f32"
    tt = torch.float32 if f32 else torch.float64
    sp = S.SimSpec(n=tuple(s["n"]), dtype=S.KH_F32 if f32 else S.KH_F64, delta=(DELTA,) * 3, dt=DT,
                   pml_lo=tuple(s["lo"]), pml_hi=tuple(s["hi"]), eps_inv=s["eps_inv"], periodic=case["periodic"])
    for a in range(3):
        sp.sigma_b[a] = s["sigma"][a]
        sp.sigma_d[a] = s["sigma"][a].copy()
    for kind, arrs in ((S.MAT_EPS_INV, s["eps"]), (S.MAT_MU_INV, s["mu"])):
        if arrs is not None:
            for c in range(3):
                sp.materials.append((kind, c, _host(arrs[c], tt)))
    if s["chi3"] is not None:
        sp.materials.append((S.MAT_CHI3, 0, _host(s["chi3"], tt)))
    for p in s["poles"]:
        sp.poles.append(S.PoleSpec(coeffs=p["coeffs"], sigma=_host(p["sigma"], torch.float64)))
    for q in s["sources"]:
        sp.sources.append(S.SourceSpec(component=q["comp"], start=tuple(q["start"]), dims=q["amp"].shape,
                                       amp=q["amp"].astype(np.complex128),
                                       time_kind=S.TIME_TABLE if "table" in q else S.TIME_GAUSSIAN, fcen=q["fcen"],
                                       width=q["width"], peak_time=q["peak"], cutoff=q["cutoff"],
                                       table=q["table"].astype(np.complex128) if "table" in q else None))
    for m in s["monitors"]:
        sp.monitors.append(S.MonitorSpec(component=m["comp"], start=tuple(m["start"]), dims=tuple(m["dims"]),
                                         freqs=m["freqs"], decimation=m["dec"]))
    for h in s["histories"]:
        sp.histories.append(S.HistorySpec(component=h["comp"], start=tuple(h["start"]), dims=tuple(h["dims"]),
                                          capacity=case["steps"]))
    return sp


def prepare(case, seed):
    _package()
    from khronos_gb300.device import GpuSim

    kind = case["kind"]
    if kind == "serve":
        cases = _serve_cases(case)
        made = [_inputs(c, seed + 101 * i) for i, c in enumerate(cases)]
        return dict(case=case, specs=[_spec(c, s) for c, s in zip(cases, made)], steps=[c["steps"] for c in cases],
                    planes=[s["planes"] for s in made])
    if kind == "gradient":
        fwd, adj = _gradient_inputs(case, seed)
        return dict(case=case, fwd=GpuSim(_spec(case, fwd)), adj=GpuSim(_spec(case, adj)),
                    dims=tuple(fwd["histories"][0]["dims"]))
    s = _inputs(case, seed)
    sp = _spec(case, s)
    st = dict(case=case, spec=sp, planes=s["planes"])
    if kind != "new":
        st["sim"] = GpuSim(sp)
    return st


def _single(case, a):
    """Values of an FP32 run in the precision they have."""
    a = np.asarray(a)
    if case["dtype"] != "f32":
        return a
    return a.astype(np.complex64 if a.dtype.kind == "c" else np.float32)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "serve":
        from khronos_gb300.serve import run_batch_concurrent

        return [[_single(case, d) for d in got] for got in
                run_batch_concurrent(state["specs"], state["steps"],
                                     collect=lambda g: [g.flux([0, 1, 2, 3], 0, DELTA * DELTA)], budget_bytes=60 << 30)]
    if kind == "gradient":
        fwd, adj, n = state["fwd"], state["adj"], case["steps"]
        fwd.reset()
        fwd.step(n)
        adj.reset()
        adj.step(n)
        grad = np.zeros(state["dims"])
        fwd.history_correlate([0, 1, 2], adj, [0, 1, 2], n, -1.0, grad)
        return {"gradient": _single(case, grad), "forward": [fwd.field_view(c) for c in range(6)]}
    if kind == "new":
        from khronos_gb300.device import GpuSim

        g = GpuSim(state["spec"])
        g.step(case["steps"])
        out = {"fields": [_single(case, g.field(c)) for c in range(6)],
               "dft": [_single(case, g.dft(m)) for m in range(len(state["spec"].monitors))]}
        g.close()
        return out
    g = state["sim"]
    g.reset()
    if kind == "watch":
        dec = state["spec"].monitors[0].decimation
        norms = []
        for ts in range(case["steps"]):
            g.step(1)
            if ts % dec == 0:
                norms.append(g.dft_norms())
        return {"norms": _single(case, np.array(norms)), "fields": [g.field_view(c) for c in range(6)]}
    g.step(case["steps"])
    return {"flux": [_single(case, g.flux(ids, axis, dA)) for ids, axis, dA in state["planes"]],
            "fields": [g.field_view(c) for c in range(6)]}


# --------------------------------------------------------------------------
# the same in 64 bits, with torch alone

STAGGER = [(0, 1, 1), (1, 0, 1), (1, 1, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1)]


class _Reference:
    """The discrete equations in FP64: fields with a ring of one cell, every
    cell through the complete cascade (σ = 0 outside the absorber)."""

    def __init__(self, case, s):
        self.case, self.s = case, s
        n = self.n = s["n"]
        dev = self.dev = _dev()
        z = lambda: torch.zeros((n[2], n[1], n[0]), device=dev, dtype=torch.float64)  # noqa: E731
        ring = lambda: torch.zeros((n[2] + 2, n[1] + 2, n[0] + 2), device=dev, dtype=torch.float64)  # noqa: E731
        self.E, self.H = [ring() for _ in range(3)], [ring() for _ in range(3)]
        self.pml = [s["lo"][a] + s["hi"][a] > 0 for a in range(3)]
        self.sig = []
        for a in range(3):
            shape = [1, 1, 1]
            shape[2 - a] = n[a]
            self.sig.append(torch.tensor(s["sigma"][a], device=dev).reshape(shape))
        self.t = [[z() for _ in range(3)] for _ in range(2)]
        self.u = [[z() if self.pml[(c + 1) % 3] else None for c in range(3)] for _ in range(2)]
        self.w = [[z() if self.pml[c] else None for c in range(3)] for _ in range(2)]
        self.P = [[[z() for _ in range(3)] for _ in range(2)] for _ in s["poles"]]
        self.F = [torch.zeros((len(m["freqs"]),) + tuple(m["dims"][::-1]), device=dev, dtype=torch.complex128)
                  for m in s["monitors"]]
        self.hist = [torch.zeros((case["steps"],) + tuple(h["dims"][::-1]), device=dev, dtype=torch.float64)
                     for h in s["histories"]]
        self.norms = []
        self.last = max(q["cutoff"] for q in s["sources"])
        self.active = True

    def inner(self, f, d=(0, 0, 0)):
        n = self.n
        return f[1 + d[2]:1 + d[2] + n[2], 1 + d[1]:1 + d[1] + n[1], 1 + d[0]:1 + d[0] + n[0]]

    def diff(self, f, axis, step):
        d = [0, 0, 0]
        d[axis] = step
        return self.inner(f, d) - self.inner(f)

    def factor(self, q, ts, h):
        t = ts * DT + (0.0 if h else DT / 2)
        if "table" in q:
            return q["table"][ts][0 if h else 1] if t <= q["cutoff"] else 0.0
        tt = t - q["peak"]
        if tt > q["cutoff"]:
            return 0.0
        return math.exp(-tt * tt / (2 * q["width"] ** 2)) * math.cos(2 * math.pi * q["fcen"] * tt)

    def half(self, h, ts):
        s, n = self.s, self.n
        A, O = (self.E, self.H) if h else (self.H, self.E)
        step = 1 if h else -1
        t, u, w = self.t[0 if h else 1], self.u[0 if h else 1], self.w[0 if h else 1]
        cd = DT / DELTA
        K = []
        for c in range(3):
            b, e = (c + 1) % 3, (c + 2) % 3
            # H: ΔB = −curl E; E: ΔD = curl H; the sign is folded into the difference's direction
            k = self.diff(A[b], e, step)
            k -= self.diff(A[e], b, step)
            K.append(k.mul_(cd))
        mats = s["mu"] if h else s["eps"]
        mc = 1.0 if h else s["eps_inv"]
        S = {}
        if self.active:
            for q in s["sources"]:
                if (q["comp"] >= 3) == h:
                    f = self.factor(q, ts, h)
                    S.setdefault(q["comp"] % 3, []).append((q, f))
        for c in range(3):
            b, e = (c + 1) % 3, (c + 2) % 3
            k = K[c]
            if self.pml[b]:
                un = ((1 - self.sig[b]) * u[c]).add_(k).div_(1 + self.sig[b])
                k = un - u[c]
                u[c] = un
            if self.pml[e]:
                t[c].mul_(1 - self.sig[e]).add_(k).div_(1 + self.sig[e])
            else:
                t[c].add_(k)
            net = t[c]
            if c in S or (not h and self.P):
                net = net.clone()
                for q, f in S.get(c, []):
                    st, dm = q["start"], q["amp"].shape
                    net[st[2]:st[2] + dm[2], st[1]:st[1] + dm[1], st[0]:st[0] + dm[0]] += \
                        f * torch.tensor(q["amp"].transpose(2, 1, 0).copy(), device=self.dev)
                if not h:
                    for P in self.P:
                        net -= P[0][c]
            wn = net * (mats[c] if mats is not None else mc)
            out = wn
            if self.pml[c]:
                out = torch.where(self.sig[c] != 0, self.inner(O[c]) + (1 + self.sig[c]) * wn - (1 - self.sig[c]) * w[c], wn)
                w[c] = wn
            self.inner(O[c]).copy_(out)
        for a in range(3):  # periodic axes: the ghost layers of the group just updated
            if (self.case["periodic"] >> a) & 1:
                for f in O:
                    v = [self.inner(f).movedim(2 - a, 0), None]
                    d = [0, 0, 0]
                    d[a] = 1
                    hi_, lo_ = v[0][n[a] - 1].clone(), v[0][0].clone()
                    self.inner(f, d).movedim(2 - a, 0)[n[a] - 1].copy_(lo_)
                    d[a] = -1
                    self.inner(f, d).movedim(2 - a, 0)[0].copy_(hi_)
        if not h:
            if s["chi3"] is not None:
                sq = sum(self.inner(O[c]) ** 2 for c in range(3))
                corr = 1.0 / (1.0 + s["chi3"] * sq)
                for c in range(3):
                    self.inner(O[c]).mul_(corr)
            for p, P in zip(s["poles"], self.P):
                co = p["coeffs"]
                drive = co["drude_coeff"] if co["is_drude"] else co["sigma_omega0_dt_sq"]
                cp = 2.0 if co["is_drude"] else 2.0 - co["omega0_dt_sq"]
                for c in range(3):
                    new = co["gamma1_inv"] * (cp * P[0][c] - co["gamma1"] * P[1][c] + drive * p["sigma"] * self.inner(O[c]))
                    new = torch.where(p["sigma"] != 0, new, P[0][c])
                    P[1][c], P[0][c] = P[0][c], new

    def box(self, comp, start, dims):
        f = (self.E + self.H)[comp]
        return f[1 + start[2]:1 + start[2] + dims[2], 1 + start[1]:1 + start[1] + dims[1],
                 1 + start[0]:1 + start[0] + dims[0]]

    def dft(self, h, ts):
        t = ts * DT + (0.0 if h else DT / 2)
        for m, F in zip(self.s["monitors"], self.F):
            if (m["comp"] >= 3) != h or ts % m["dec"]:
                continue
            ph = torch.tensor(DT * np.exp(2j * math.pi * m["freqs"] * t), device=self.dev)
            F += ph[:, None, None, None] * self.box(m["comp"], m["start"], m["dims"])[None]

    def run(self, steps, norms=False):
        for ts in range(steps):
            if self.active and ts * DT > self.last:
                self.active = False
            self.half(True, ts)
            self.dft(True, ts)
            self.half(False, ts)
            self.dft(False, ts)
            for h, buf in zip(self.s["histories"], self.hist):
                buf[ts] = self.box(h["comp"], h["start"], h["dims"])
            if norms and ts % self.s["monitors"][0]["dec"] == 0:
                self.norms.append([float(torch.linalg.vector_norm(F)) for F in self.F])
        return self

    def fields(self):
        """The component arrays with their staggered layers, indexed [i, j, k]."""
        out = []
        for c, f in enumerate(self.E + self.H):
            d = [self.n[a] + STAGGER[c][a] for a in range(3)]
            out.append(f[1:1 + d[2], 1:1 + d[1], 1:1 + d[0]].permute(2, 1, 0))
        return out

    def flux(self, ids, axis, dA):
        e1, e2, h1, h2 = [self.F[i] for i in ids]
        return ((e1 * h2.conj()).real - (e2 * h1.conj()).real).sum(dim=(1, 2, 3)).mul(dA).cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind == "serve":
        out = []
        for i, c in enumerate(_serve_cases(case)):
            s = _inputs(c, seed + 101 * i)
            out.append([_Reference(c, s).run(c["steps"]).flux([0, 1, 2, 3], 0, DELTA * DELTA)])
        return out
    if kind == "gradient":
        fwd, adj = [_Reference(case, s).run(case["steps"]) for s in _gradient_inputs(case, seed)]
        g = sum((f * a.flip(0)).sum(dim=0) for f, a in zip(fwd.hist, adj.hist))
        return {"gradient": (-g).permute(2, 1, 0), "forward": fwd.fields()}
    s = _inputs(case, seed)
    r = _Reference(case, s).run(case["steps"], norms=kind == "watch")
    if kind == "watch":
        return {"norms": np.array(r.norms), "fields": r.fields()}
    if kind == "new":
        return {"fields": r.fields(), "dft": [F.permute(3, 2, 1, 0) for F in r.F]}
    return {"flux": [r.flux(*p) for p in s["planes"]], "fields": r.fields()}


# --------------------------------------------------------------------------
# what a pass cannot do without

def _work(case, monitors):
    n = (case["nx"], case["ny"], case["nz"])
    cells = n[0] * n[1] * n[2]
    size = 4 if case["dtype"] == "f32" else 8
    lo, hi = _widths(case)
    inside = [(lo[a] + hi[a]) / n[a] for a in range(3)]
    # per cell and step: six fields read and written once, the per-voxel materials read
    words = 12.0 + (3 if case["voxel"] else 0) + (3 if case["mu"] else 0)
    # absorber: one auxiliary per half for the component along the axis, one where two axes meet
    words += 4 * sum(inside)
    words += 4 * (inside[0] * inside[1] + inside[1] * inside[2] + inside[2] * inside[0])
    flops = 36.0 + 12 * sum(inside)
    if case["chi3"]:
        words += 1 * 0.16
        flops += 10 * 0.16
    if case["poles"]:
        ball = case["poles"] * 4 * 4.19 * (0.12 * min(n)) ** 3 / cells
        words += 13 * ball
        flops += 24 * ball
    b = cells * case["steps"] * words * size
    f = cells * case["steps"] * flops
    for items, dec in monitors:
        updates = math.ceil(case["steps"] / dec)
        b += updates * items * 2 * size * (4 if size == 4 else 2)
        f += updates * items * (10 if size == 4 else 4)
    return b, f


def _monitor_items(case):
    n = (case["nx"], case["ny"], case["nz"])
    lo, hi = _widths(case)
    normal = 2 if case["periodic"] & 1 else 0
    dims = [1 if a == normal else max(1, n[a] - lo[a] - hi[a] - 2) for a in range(3)]
    dec = max(1, int(1.0 / (2 * FCEN * 1.25 * DT) / 4))
    planes = 2 if case["source"] == "plane" else 1
    return [(dims[0] * dims[1] * dims[2] * case["nf"], dec)] * (4 * planes)


def work(case):
    kind = case["kind"]
    if kind == "serve":
        got = [_work(c, _monitor_items(c)) for c in _serve_cases(case)]
        return {"bytes": sum(g[0] for g in got), "flops": sum(g[1] for g in got)}
    if kind == "gradient":
        b, f = _work(case, [])
        n = (case["nx"], case["ny"], case["nz"])
        voxels = max(2, int(0.3 * n[0])) * max(2, int(0.3 * n[1])) * max(2, int(0.18 * n[2]))
        per = voxels * 3 * case["steps"]
        return {"bytes": 2 * b + per * 4 * 4, "flops": 2 * f + per * 2}
    b, f = _work(case, _monitor_items(case))
    if kind == "new":  # the materials come from the host, the fields and DFT arrays go back
        cells = case["nx"] * case["ny"] * case["nz"]
        b += cells * 4 * 3 + cells * 4 * 6 + sum(i for i, _ in _monitor_items(case)) * 8
    return {"bytes": b, "flops": f}
