"""What a user of the stepper has it do, as cases that can be timed.

The sizes are those of this repository's configurations: the 64^3 junction (and the 65^3 that the
reference's grid rounding gives for the same cell), the 96-member CEP/amplitude sweep over 96^3, 128^3
and 192^3, the bowtie, the Au-on-quartz inverse design and the 160^3 adjoint case, and what follows a run:
phases, spectra, and the rasteriser before it.  draw() spreads sizes, precisions and options over the
same ranges.

A stepping case keeps a Fields in mid-run, as a program does that steps and reads its monitors in turn;
a pass advances it by `steps` steps.  A job is a whole run from descriptors to read-back.
"""
import math

import numpy as np
import torch

from sim_juncs_gb300 import _abi
from sim_juncs_gb300.configs import AU, QUARTZ, bowtie_instance, stable_courant
from sim_juncs_gb300.geometry import Box, Union
from sim_juncs_gb300.spec import (PML, Design, Grid, Instance, Objective, Probe, Region, Scene, Source,
                                  Susceptibility)

SAVE_SPAN = 20
FCEN = 1 / 0.7


def listed():
    return [
        # the smallest whole run: the 64^3 junction of the plain method, default precision, 2000 steps
        dict(name="job_junction64_f64", kind="job", nx=64, ny=64, nz=64, res=20.0, scene="au", prec="f64",
             count=1, steps=2000, dft=True, graph=0),
        # the same junction in FP32, stepping on and reading its monitors (launches and latency count)
        dict(name="step_junction64_f32", kind="step", nx=64, ny=64, nz=64, res=20.0, scene="au", prec="f32",
             count=1, steps=500, warm=60, dft=True, graph=0),
        # the grid the reference's rounding gives (odd rows), default precision, replayed as graphs
        dict(name="step_junction65_f64", kind="step", nx=65, ny=65, nz=65, res=65 / 3.2, scene="au", prec="f64",
             count=1, steps=500, warm=60, dft=True, graph=50),
        # the CEP/amplitude sweep: 32 members each at 96^3, 128^3 and 192^3, one batch
        dict(name="step_sweep96_f32", kind="sweep", per_size=32, prec="f32", steps=20, warm=160, graph=5),
        # production bowtie: 512 x 512 x 384, Ez plane, 50-frequency DFTs
        dict(name="step_bowtie_f32", kind="bowtie", nx=512, ny=512, nz=384, res=40.0, prec="f32", steps=20,
             warm=160, graph=0),
        # the bowtie's cell at half the resolution in FP64 (the plain path)
        dict(name="step_bowtie256_f64", kind="bowtie", nx=256, ny=256, nz=192, res=20.0, prec="f64", steps=40,
             warm=100, graph=0),
        # forward steps of the inverse-design batch: half of every grid is dispersive quartz
        dict(name="step_quartz192x4_f32", kind="step", nx=192, ny=192, nz=192, res=30.0, scene="quartz",
             prec="f32", count=4, steps=20, warm=100, dft=False, graph=0),
        # one gradient of the adjoint case through torch.autograd
        dict(name="adjoint160_f32", kind="autograd", n=160, res=30.0, scene="au", prec="f32", design=18, thick=3,
             steps=200, every=100),
        # one iteration of the batched inverse design (fewer designs and steps)
        dict(name="inverse192x4_f32", kind="inverse", n=192, res=30.0, scene="quartz", prec="f32", design=24,
             thick=3, count=4, steps=60, every=30),
        # CEP and envelope of a sweep's 96 x 4 gap series of 200 samples
        dict(name="phases_sweep", kind="phases", series=384, samples=200),
        # spectra of a 32 x 32 monitor plane after a run of 1000 samples
        dict(name="spectrum_plane", kind="spectrum", plane=32, samples=1000, n=48, prec="f32"),
        # the rasteriser on the bowtie's scene
        dict(name="raster_bowtie256", kind="raster", nx=256, ny=256, nz=192, res=20.0, scene="bowtie", smooth=0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step"] * 4 + ["job", "sweep", "bowtie", "autograd", "inverse", "phases", "spectrum", "raster"])
    prec = rng.choice(["f32", "f32", "f64"])
    if kind in ("step", "job"):
        scene = rng.choice(["au", "au", "quartz"])
        lo, hi = (48 if scene == "quartz" else 36), (96 if kind == "job" else 256)
        nx, ny, nz = (_log(rng, lo, hi) for _ in range(3))
        if rng.random() < 0.5:
            nx = max(64, nx // 32 * 32)
        count = rng.choice([1, 1, 2, 5])
        steps = max(20, min(2000 if kind == "job" else 500, int(4e8 / (nx * ny * nz * count))))
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, scene=scene, prec=prec, count=count, steps=steps,
                    # quartz's Lorentz term at 10 / um needs the finer time steps
                    res=30.0 if scene == "quartz" else rng.choice([20.0, 30.0, 40.0]),
                    warm=0 if kind == "job" else 60, dft=rng.random() < 0.5,
                    graph=0 if rng.random() < 0.6 else rng.choice([5, 10, 25]))
    if kind == "sweep":
        return dict(kind=kind, per_size=_log(rng, 1, 16), prec=prec, steps=rng.randint(8, 16), warm=160,
                    graph=rng.choice([0, 5]))
    if kind == "bowtie":
        return dict(kind=kind, nx=_log(rng, 160, 400), ny=_log(rng, 160, 400), nz=_log(rng, 120, 300),
                    res=rng.choice([16.0, 20.0]), prec=prec, steps=20, warm=100, graph=0)
    if kind in ("autograd", "inverse"):
        n = _log(rng, 40, 150)
        return dict(kind=kind, n=n, res=30.0, scene=rng.choice(["au", "quartz"]), prec=prec,
                    design=rng.randint(6, 20), thick=rng.randint(1, 3), count=1 if kind == "autograd" else rng.randint(2, 3),
                    steps=rng.randint(60, 120), every=rng.choice([30, 50, 1000]))
    if kind == "phases":
        return dict(kind=kind, series=_log(rng, 1, 1500), samples=_log(rng, 96, 600))
    if kind == "spectrum":
        return dict(kind=kind, plane=_log(rng, 2, 32), samples=_log(rng, 20, 1500), n=_log(rng, 36, 64), prec=prec)
    return dict(kind=kind, nx=_log(rng, 64, 256), ny=_log(rng, 64, 256), nz=_log(rng, 64, 192), res=20.0,
                scene=rng.choice(["au", "quartz", "bowtie"]), smooth=rng.choice([0, 0, 1]))


# ------------------------------------------------------------------ scenes
def _pml(nx, ny, nz, dx):
    return min(0.5, 0.16 * min(nx, ny, nz) * dx)


def _boxes(nx, ny, nz, dx, scene, shift=0.0):
    """Regions of the junction as (boxes, eps, poles): Au box pair, then the quartz substrate."""
    cx, cy, cz = nx * dx / 2, ny * dx / 2, nz * dx / 2
    gap, by, bz = 0.2 + shift, 0.5 + shift, 0.1
    bx = min(1.0, cx - gap / 2 - _pml(nx, ny, nz, dx))  # the gold ends where the absorber begins, as in the 3.2 um cell
    au = [((cx - gap / 2 - bx, cy - by / 2, cz - bz / 2), (cx - gap / 2, cy + by / 2, cz + bz / 2)),
          ((cx + gap / 2, cy - by / 2, cz - bz / 2), (cx + gap / 2 + bx, cy + by / 2, cz + bz / 2))]
    regions = [(au, 1.0, AU)]
    if scene == "quartz":
        regions.append(([((0.0, 0.0, 0.0), (nx * dx, ny * dx, cz - bz / 2))], 2.1, QUARTZ))
    return regions


def _scene(regions, smooth=0):
    rs = [Region(Union(*[Box(a, b) for a, b in boxes]) if len(boxes) > 1 else Box(*boxes[0]), eps=eps,
                 susceptibilities=[Susceptibility(s.omega_0, s.gamma, s.sigma, s.drude) for s in poles])
          for boxes, eps, poles in regions]
    return Scene(rs, 1.0, _abi.EPS_SUM if smooth else _abi.EPS_FIRST, smooth_n=smooth)


def _pulse(rng, Lx, Ly, z):
    """An x-polarised sheet whose pulse is well on its way at t = 0; CEP and amplitude as a sweep draws them."""
    phase, amp = float(rng.uniform(0, 2 * math.pi)), float(10 ** rng.uniform(-1, 1))
    return Source(_abi.EX, FCEN, 2.0, -9.0, 11.0, (0.0, 0.0, z), (Lx, Ly, z), phase=phase, amplitude=amp)


def _junction(rng, nx, ny, nz, res, scene, comps, dft):
    dx = 1.0 / res
    dt = stable_courant(res) * dx
    cx, cy, cz = nx * dx / 2, ny * dx / 2, nz * dx / 2
    pml = _pml(nx, ny, nz, dx)
    src = _pulse(rng, nx * dx, ny * dx, cz - min(1.0, 0.5 * (cz - pml)))
    probes = [Probe(_abi.COMPONENTS[c], (cx + d, cy, cz), monitor=True, dft=dft)
              for c in comps for d in (-0.075, -0.025, 0.025, 0.075)]
    freqs = [0.9 * FCEN, FCEN, 1.1 * FCEN] if dft else []
    return Instance(Grid(nx, ny, nz, dx, dt), _scene(_boxes(nx, ny, nz, dx, scene)), PML(pml), [src], probes, freqs,
                    SAVE_SPAN)


def _instances(case, seed):
    rng = np.random.default_rng(seed)
    if case["kind"] == "sweep":
        return [_junction(rng, n, n, n, res, "au", ("Ez",), False)
                for n, res in ((96, 30.0), (128, 40.0), (192, 60.0)) for _ in range(case["per_size"])]
    if case["kind"] == "bowtie":
        inst = bowtie_instance(case["nx"], case["ny"], case["nz"], case["res"])
        s = inst.sources[0]
        g = inst.grid
        inst.sources = [_pulse(rng, g.nx * g.dx, g.ny * g.dx, s.lo[2])]
        inst.sources[0].frequency = 1 / 0.8
        return [inst]
    return [_junction(rng, case["nx"], case["ny"], case["nz"], case["res"], case["scene"], ("Ex", "Ez"), case["dft"])
            for _ in range(case["count"])]


def _designs(case, seed):
    """Per design: (instance, lo, eps on the GPU, objective) of the adjoint cases."""
    rng = np.random.default_rng(seed)
    n, nd, th = case["n"], case["design"], case["thick"]
    m = n // 2
    out = []
    for _ in range(case.get("count", 1)):
        inst = _junction(rng, n, n, n, case["res"], case["scene"], ("Ex",), False)
        lo = (m - nd // 2, m - nd // 2, m - th // 2)
        eps = torch.from_numpy(rng.uniform(1.0, 4.0, size=(th, nd, nd)))
        cells = np.array([[m - 2 + a, m - 2 + b, m] for b in range(5) for a in range(5)])
        out.append((inst, lo, eps.to("cuda", torch.float64 if case["prec"] == "f64" else torch.float32),
                    Objective(cells, frequency=FCEN, comps=(0, 1, 2))))
    return out


def _series(case, seed):
    """Gap-like pulses: a Gaussian envelope on a carrier that the sampling resolves, per series its own CEP,
    amplitude, centre and width, over a slow background as near-field monitors have."""
    rng = np.random.default_rng(seed)
    n, m = case["series"], case["samples"]
    t = np.arange(m) * 0.1
    T = t[-1]
    f0 = rng.uniform(1.2, 1.8, (n, 1))
    t0 = rng.uniform(0.42, 0.58, (n, 1)) * T
    sig = rng.uniform(0.7, 1.1, (n, 1))
    v = 10 ** rng.uniform(-1, 1, (n, 1)) * np.exp(-0.5 * ((t - t0) / sig) ** 2) * np.cos(
        2 * np.pi * f0 * (t - t0) + rng.uniform(0, 2 * np.pi, (n, 1)))
    return t, v


def _bowtie_scene(case, rng):
    inst = bowtie_instance(case["nx"], case["ny"], case["nz"], case["res"])
    inst.material.regions[1].obj = Box((0.0, 0.0, 1.0 + float(rng.uniform(0, 1))),
                                       (case["nx"] / case["res"], case["ny"] / case["res"],
                                        case["nz"] / case["res"] / 2 - float(rng.uniform(0.1, 1))))
    return inst.grid, inst.material


# ------------------------------------------------------------------ the passes
def prepare(case, seed):
    from sim_juncs_gb300.fields import Fields
    kind = case["kind"]
    if kind == "job":
        return dict(case=case, insts=_instances(case, seed))
    if kind in ("step", "sweep", "bowtie"):
        f = Fields(_instances(case, seed), case["prec"])
        f.step(case["warm"])
        f.synchronize()
        return dict(case=case, f=f)
    if kind in ("autograd", "inverse"):
        ds = _designs(case, seed)
        return dict(case=case, f=Fields([d[0] for d in ds], case["prec"]), designs=ds)
    if kind == "phases":
        t, v = _series(case, seed)
        return dict(case=case, t=t, v=v)
    if kind == "spectrum":
        f = Fields(_plane(case, seed), case["prec"])
        f.step(case["samples"])
        f.synchronize()
        return dict(case=case, f=f)
    rng = np.random.default_rng(seed)
    if case["scene"] == "bowtie":
        grid, scene = _bowtie_scene(case, rng)
        if case["smooth"]:
            scene = Scene(scene.regions, 1.0, _abi.EPS_SUM, smooth_n=case["smooth"])
    else:
        dx = 1.0 / case["res"]
        grid = Grid(case["nx"], case["ny"], case["nz"], dx)
        scene = _scene(_boxes(case["nx"], case["ny"], case["nz"], dx, case["scene"], float(rng.uniform(0, 0.7))),
                       case["smooth"])
    return dict(case=case, grid=grid, scene=scene)


def _plane(case, seed):
    """A junction whose monitors are a plane of Ez points, sampled on every step."""
    inst = _junction(np.random.default_rng(seed), case["n"], case["n"], case["n"], 20.0, "au", (), False)
    g, p = inst.grid, case["plane"]
    c, d = g.nx * g.dx / 2, min(g.dx, 0.5 * g.nx * g.dx / p)
    inst.probes = [Probe(_abi.EZ, (c + (a - p / 2) * d, c + (b - p / 2) * d, c)) for b in range(p) for a in range(p)]
    inst.save_span = 1
    return inst


def _step(f, case):
    if case["graph"]:
        f.step_graph(case["steps"], case["graph"])
    else:
        f.step(case["steps"])
    return {"monitors": [f.monitors(q) for q in range(f.n_instances)] if f.n_instances <= 8
            else np.concatenate([f.monitors(q) for q in range(f.n_instances)]),
            "dft": [f.dft(q) for q in range(f.n_instances) if f.instances[q].n_dft]}


def run(state):
    from sim_juncs_gb300.fields import Fields, rasterize, rasterize_counts
    case = state["case"]
    kind = case["kind"]
    if kind == "job":
        with Fields(state["insts"], case["prec"]) as f:
            return _step(f, case)
    if kind in ("step", "sweep", "bowtie"):
        return _step(state["f"], case)
    if kind == "autograd":
        from sim_juncs_gb300.autograd import GapFieldObjective
        _, lo, eps, ob = state["designs"][0]
        e = eps.clone().requires_grad_(True)
        F = GapFieldObjective.apply(e, state["f"], lo, ob, case["steps"], case["every"])
        F.backward()
        return {"F": F.detach(), "grad": e.grad}
    if kind == "inverse":
        f, ds = state["f"], state["designs"]
        for q, (_, lo, eps, _) in enumerate(ds):
            f.set_design(Design(lo, eps.cpu().numpy()), q)
        F, grads = f.adjoint_gradient([d[3] for d in ds], case["steps"], case["every"])
        return {"F": F, "grad": [torch.from_numpy(g).to(d[2]) for g, d in zip(grads, ds)]}
    if kind == "phases":
        from sim_juncs_gb300.phases import extract_phases
        res = extract_phases(state["t"], state["v"], 2.0)
        out = {k: np.array([r[k] for r in res]) for k in ("f0", "phi", "t0_corr", "t0", "mu", "sig", "skew", "amp")}
        out["bins"] = np.array([[r[k] for k in ("f0_ind", "band_lo", "band_hi", "lowpass_steps", "status")] for r in res])
        return out
    if kind == "spectrum":
        return state["f"].monitor_spectrum()
    return (rasterize_counts if case["smooth"] else rasterize)(state["grid"], state["scene"])


def work(case):
    kind = case["kind"]
    s = 8 if case.get("prec") == "f64" else 4

    def voxel_bytes(nx, ny, nz, res, pml, quartz):
        # per step: 6 components read and written and the material byte; 2 psi per E and H and slab axis
        # read and written; P^n, P^{n-1} of the poles read and P^{n+1}, P^n written
        slab = sum(min(1.0, 2 * pml * res / n) for n in (nx, ny, nz))
        au = 2 * (1.0 * 0.5 * 0.1) * res ** 3
        return nx * ny * nz * (12.0 * s + 1 + slab * 8 * s + (0.5 * 12 * s if quartz else 0)) + au * 2 * 12 * s

    def junction(nx, ny, nz, res, quartz=False):
        return voxel_bytes(nx, ny, nz, res, min(0.5, 0.16 * min(nx, ny, nz) / res), quartz)

    if kind in ("step", "job"):
        b = case["steps"] * case["count"] * junction(case["nx"], case["ny"], case["nz"], case["res"], case["scene"] == "quartz")
        v = case["steps"] * case["count"] * case["nx"] * case["ny"] * case["nz"]
    elif kind == "sweep":
        b = case["steps"] * case["per_size"] * sum(junction(n, n, n, r) for n, r in ((96, 30.0), (128, 40.0), (192, 60.0)))
        v = case["steps"] * case["per_size"] * (96 ** 3 + 128 ** 3 + 192 ** 3)
    elif kind == "bowtie":
        v = case["nx"] * case["ny"] * case["nz"] * case["steps"]
        b = case["steps"] * (voxel_bytes(case["nx"], case["ny"], case["nz"], case["res"], 1.0, False) + 4096 * 50 * 32)
    elif kind in ("autograd", "inverse"):
        # forward twice (once to the objective, once again for the gradient), then the transposed step
        c, n = case.get("count", 1), case["n"]
        b = 3 * case["steps"] * c * junction(n, n, n, case["res"], case["scene"] == "quartz")
        v = 3 * case["steps"] * c * n ** 3
    elif kind == "phases":
        b, n = case["series"] * (case["samples"] * 8 + 120.0), case["samples"]
        return {"bytes": b, "flops": case["series"] * 3 * 5.0 * n * math.log2(n)}
    elif kind == "spectrum":
        np2, m = 2 ** int(math.log2(case["samples"])), case["plane"] ** 2
        return {"bytes": m * (case["samples"] * 8 + np2 * 16.0), "flops": m * 5.0 * np2 * max(1.0, math.log2(np2))}
    else:
        v = case["nx"] * case["ny"] * case["nz"]
        return {"bytes": 3.0 * v, "flops": 3.0 * v * 30}
    return {"bytes": float(b), "flops": 24.0 * v}


# ------------------------------------------------------------------ the same in 64 bits, plain torch
class _Exact:
    """The leapfrog of one instance in FP64: arrays [nz][ny][nx], CPML auxiliaries on the whole grid
    (b = 1, c = 0 outside the absorber), ADE polarisations, the sheet source, trilinear probes."""

    OFF = ((.5, 0, 0), (0, .5, 0), (0, 0, .5), (0, .5, .5), (.5, 0, .5), (.5, .5, 0))

    def __init__(self, inst, inside, regions, design=None):
        g = self.g = inst.grid
        self.dx, self.dt, self.S = g.dx, g.dt, g.dt / g.dx
        self.shape = (g.nz, g.ny, g.nx)
        self.n = (g.nx, g.ny, g.nz)
        k = dict(dtype=torch.float64, device="cuda")
        self.k = k
        ax = [torch.arange(m, **k) for m in self.n]
        self.einv, self.poles = [], []
        for c in range(3):
            x = [(ax[a] + self.OFF[c][a]) * g.dx for a in range(3)]
            x = (x[0].view(1, 1, -1), x[1].view(1, -1, 1), x[2].view(-1, 1, 1))
            free = torch.ones(self.shape, dtype=torch.bool, device="cuda")
            eps = torch.ones(self.shape, **k)
            here = []
            for (eps_r, poles), f in zip(regions, inside):
                hit = f(*x).expand(self.shape) & free
                free = free & ~hit
                eps = torch.where(hit, torch.full_like(eps, eps_r), eps)
                here.append(hit)
            self.einv.append(1.0 / eps)
            row = []
            for (_, poles), hit in zip(regions, here):
                for p in poles:
                    w, gm = 2 * math.pi * p.omega_0, 2 * math.pi * p.gamma
                    den = 1 + gm * self.dt / 2
                    A = (2 - (0.0 if p.drude else w * w * self.dt ** 2)) / den
                    row.append((A, -(1 - gm * self.dt / 2) / den, w * w * self.dt ** 2 / den * p.sigma * hit.double()))
            self.poles.append(row)
        d = inst.pml.thickness
        self.prof = []
        for a in range(3):
            L = self.n[a] * g.dx
            out = []
            for h in (0.0, 0.5):
                q = (ax[a] + h) * g.dx
                u = torch.clamp(torch.maximum((d - q) / d, (q - (L - d)) / d), min=0.0)
                s = -3 * math.log(1e-15) / (2 * d) * u ** 2
                b = torch.exp(-s * self.dt)
                out.append([v.view([-1 if z == 2 - a else 1 for z in range(3)]) for v in (b, b - 1.0)])
            # c = s/(s + alpha) (b - 1) with alpha = 0; the other axis' points of the slab have b = 1, c = 0
            self.prof.append(out)
        z = lambda: torch.zeros(self.shape, **k)  # noqa: E731
        self.E, self.H = [z() for _ in range(3)], [z() for _ in range(3)]
        self.pE, self.pH = {}, {}
        self.P = [[(z(), z()) for _ in row] for row in self.poles]
        s = inst.sources[0]
        self.src = s
        u = s.lo[2] / g.dx
        i0, f = int(math.floor(u)), u - math.floor(u)
        w = torch.zeros(g.nz, **k)
        w[i0] += (1 - f) / g.dx
        if i0 + 1 < g.nz:
            w[i0 + 1] += f / g.dx
        wxy = []
        for a in range(2):
            q = (ax[a] + self.OFF[s.component][a]) * g.dx
            lo, hi = s.lo[a], s.hi[a]
            wxy.append(torch.clamp(torch.clamp(q + g.dx / 2, max=hi) - torch.clamp(q - g.dx / 2, min=lo), min=0.0) / g.dx)
        self.w = w.view(-1, 1, 1) * wxy[1].view(1, -1, 1) * wxy[0].view(1, 1, -1)
        self.design = design
        self.t = 0

    def dipole(self, t):
        s = self.src
        peak, cut = 0.5 * (s.start_time + s.end_time), 0.5 * (s.end_time - s.start_time)
        while math.exp(-cut * cut / (2 * s.width ** 2)) < 1e-100:
            cut *= 0.9
        tt = t - peak
        if float(np.float32(abs(tt))) > float(np.float32(cut)):
            return 0j
        om = 2 * math.pi * s.frequency
        a = -om * tt - (s.phase + math.pi)
        return math.exp(-tt * tt / (2 * s.width ** 2)) * complex(math.cos(a), math.sin(a)) / complex(0, -om)

    def _diff(self, v, a, fwd):
        d = 2 - a
        m = self.shape[d]
        zero = torch.zeros_like(v.narrow(d, 0, 1))
        if fwd:
            return torch.cat([v.narrow(d, 1, m - 1), zero], d) - v
        return v - torch.cat([zero, v.narrow(d, 0, m - 1)], d)

    def _curl(self, F, psi, half, fwd):
        out = []
        for c in range(3):
            a1, a2 = (c + 1) % 3, (c + 2) % 3
            cv = 0
            for a, o, sg in ((a1, a2, 1.0), (a2, a1, -1.0)):
                d = self._diff(F[o], a, fwd)
                b, cc = self.prof[a][half]
                p = cc * d if (c, a) not in psi else b * psi[(c, a)] + cc * d
                psi[(c, a)] = p
                cv = cv + sg * (d + p)
            out.append(cv)
        return out

    def step(self):
        cv = self._curl(self.E, self.pH, 1, True)
        self.H = [h - self.S * v for h, v in zip(self.H, cv)]
        cv = self._curl(self.H, self.pE, 0, False)
        t = (self.t + 0.5) * self.dt
        s = self.src
        J = (complex(s.amplitude) * (self.dipole(t) - self.dipole(t - self.dt))).real
        new = []
        for c in range(3):
            acc = self.S * cv[c]
            if c == s.component:
                acc = acc - J * self.w
            for p, (A, B, C) in enumerate(self.poles[c]):
                pn, pq = self.P[c][p]
                pp = A * pn + B * pq + C * self.E[c]
                acc = acc - (pp - pn)
                self.P[c][p] = (pp, pn)
            e = self.E[c] + self.einv[c] * acc
            if self.design is not None:
                (i, j, k), eps = self.design
                n2, n1, n0 = eps.shape
                box = (slice(k, k + n2), slice(j, j + n1), slice(i, i + n0))
                add = (1.0 / eps - self.einv[c][box]) * acc[box]
                e = e + torch.nn.functional.pad(add, (i, self.n[0] - i - n0, j, self.n[1] - j - n1, k, self.n[2] - k - n2))
            new.append(e)
        self.E = new
        self.t += 1

    def probe_table(self, probes):
        idx, wt, comp = [], [], []
        for p in probes:
            i0, f = [], []
            for a in range(3):
                u = p.pos[a] / self.dx - self.OFF[p.component][a]
                i0.append(int(math.floor(u)))
                f.append(u - math.floor(u))
            for m in range(8):
                q = [i0[a] + ((m >> a) & 1) for a in range(3)]
                ok = all(0 <= q[a] < self.n[a] for a in range(3))
                w = math.prod(f[a] if (m >> a) & 1 else 1 - f[a] for a in range(3))
                idx.append((q[2] * self.n[1] + q[1]) * self.n[0] + q[0] if ok else 0)
                wt.append(w if ok else 0.0)
            comp.append(p.component)
        groups = []
        comp = np.array(comp)
        for c in sorted(set(comp.tolist())):
            at = np.nonzero(comp == c)[0]
            groups.append((c, torch.from_numpy(at).cuda(), torch.tensor(np.array(idx).reshape(-1, 8)[at]).cuda(),
                           torch.tensor(np.array(wt).reshape(-1, 8)[at]).cuda()))
        return groups, torch.tensor(comp >= 3).cuda()

    def sample(self, table):
        groups, is_h = table
        out = torch.zeros(len(is_h), **self.k)
        for c, at, idx, wt in groups:
            out[at] = ((self.E + self.H)[c].reshape(-1)[idx] * wt).sum(1)
        return out


def _in_boxes(boxes):
    cs = [(tuple(a[q] + (b[q] - a[q]) / 2 for q in range(3)), tuple((b[q] - a[q]) / 2 for q in range(3))) for a, b in boxes]

    def f(x, y, z):
        r = None
        for c, o in cs:
            h = ((x - c[0]).abs() <= o[0]) & ((y - c[1]).abs() <= o[1]) & ((z - c[2]).abs() <= o[2])
            r = h if r is None else r | h
        return r
    return f


def _in_bowtie(case):
    dx = 1.0 / case["res"]
    cx, cy, cz = case["nx"] * dx / 2, case["ny"] * dx / 2, case["nz"] * dx / 2
    top, bot, Ly = cz + 0.025, cz - 0.025, case["ny"] * dx
    tan = math.tan(math.radians(30.0))
    nrm = math.sqrt(tan * tan + 1.0)

    def prisms(x, y, z):
        r = None
        for side in (-1, 1):
            tip = cx + side * 0.05
            base = tip + side * 2.0
            n0, n1 = -side * tan / nrm, 1.0 / nrm
            s = math.sqrt(n0 * n0 + n1 * n1)
            h = ((n0 / s) * x + (n1 / s) * y <= (cy - side * tan * tip) / nrm)
            h = h & ((n0 / s) * x - (n1 / s) * y <= (-cy - side * tan * tip) / nrm)
            lo, hi = (tip, base) if side > 0 else (base, tip)
            h = h & _in_boxes([((lo, 0.0, bot), (hi, Ly, top))])(x, y, z)
            r = h if r is None else r | h
        return r
    slab = _in_boxes([((0.0, 0.0, bot - 1.0), (case["nx"] * dx, Ly, bot))])
    return [prisms, slab], [(1.0, AU), (2.13, [])]


def _exact_for(inst, case, design=None):
    if case["kind"] == "bowtie":
        inside, regions = _in_bowtie(case)
    else:
        g = inst.grid
        rs = _boxes(g.nx, g.ny, g.nz, g.dx, case.get("scene", "au"))
        inside, regions = [_in_boxes(b) for b, _, _ in rs], [(e, p) for _, e, p in rs]
    return _Exact(inst, inside, regions, design)


def _exact_run(inst, case, steps):
    with torch.no_grad():
        x = _exact_for(inst, case)
        table = x.probe_table(inst.probes)
        mon = torch.tensor([p.monitor for p in inst.probes]).cuda()
        dft = torch.tensor([p.dft for p in inst.probes]).cuda()
        fr = torch.tensor([float(f) for f in inst.freqs], dtype=torch.float64, device="cuda")
        D = torch.zeros((len(inst.probes), len(fr)), dtype=torch.complex128, device="cuda")
        rows = []
        for n in range(steps):
            v = None
            if n % inst.save_span == 0 or len(fr):
                v = x.sample(table)
            if n % inst.save_span == 0:
                rows.append(v[mon])
            if len(fr):
                t = (n - 0.5 * table[1].double()) * x.dt
                D += x.dt * v[:, None] * torch.exp(2j * math.pi * fr[None, :] * t[:, None])
            x.step()
        return torch.stack(rows, 1).cpu().numpy(), D[dft].cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind in ("step", "job", "sweep", "bowtie"):
        insts = _instances(case, seed)
        steps = case["steps"] + (0 if kind == "job" else case["warm"])
        # a step of the plain version takes about 2 ms + 0.5 ns per voxel
        if sum(steps * (2e-3 + 5e-10 * i.grid.voxels) for i in insts) > 15:
            return None
        got = [_exact_run(i, case, steps) for i in insts]
        return {"monitors": [m for m, _ in got] if len(got) <= 8 else np.concatenate([m for m, _ in got]),
                "dft": [d for (_, d), i in zip(got, insts) if i.n_dft]}
    if kind in ("autograd", "inverse"):
        ds = _designs(case, seed)
        if len(ds) * case["steps"] * (8e-3 + 3e-9 * case["n"] ** 3) > 18:
            return None
        Fs, gs = [], []
        for inst, lo, eps, ob in ds:
            e = eps.double().requires_grad_(True)
            x = _exact_for(inst, case, (lo, e))
            at = torch.from_numpy(np.asarray(ob.cells)).cuda()
            D = 0
            for n in range(case["steps"]):
                v = torch.stack([x.E[c][at[:, 2], at[:, 1], at[:, 0]] for c in range(3)])
                a = 2 * math.pi * FCEN * n * x.dt
                D = D + x.dt * torch.stack([v * math.cos(a), v * math.sin(a)])
                x.step()
            F = (D ** 2).sum()
            F.backward()
            Fs.append(F.detach())
            gs.append(e.grad.to(eps.dtype) if kind == "autograd" else e.grad)
            del x, D, F
        if kind == "autograd":
            return {"F": Fs[0], "grad": gs[0]}
        return {"F": torch.stack(Fs).cpu().numpy(), "grad": gs}
    if kind == "spectrum":
        inst = _plane(case, seed)
        mon, _ = _exact_run(inst, case, case["samples"])
        N = mon.shape[1]
        n2 = 2 ** int(math.log(N) / math.log(2.0))
        k = np.arange(n2)
        k = np.where(k < n2 // 2, k, k - n2)
        ph = np.exp(-2j * np.pi * ((np.arange(n2)[:, None] * k[None, :]) % N) / N)
        return mon[:, :n2] @ ph
    if kind == "raster" and not case["smooth"] and case["scene"] != "bowtie":
        dx = 1.0 / case["res"]
        rs = _boxes(case["nx"], case["ny"], case["nz"], dx, case["scene"],
                    float(np.random.default_rng(seed).uniform(0, 0.7)))
        out = torch.zeros((3, case["nz"], case["ny"], case["nx"]), dtype=torch.uint8, device="cuda")
        for c in range(3):
            x = [(torch.arange(m, dtype=torch.float64, device="cuda") + _Exact.OFF[c][a]) * dx
                 for a, m in enumerate((case["nx"], case["ny"], case["nz"]))]
            for r, (boxes, _, _) in enumerate(rs):
                out[c] |= _in_boxes(boxes)(x[0].view(1, 1, -1), x[1].view(1, -1, 1), x[2].view(-1, 1, 1)).to(torch.uint8) << r
        return out.cpu().numpy()
    return None
