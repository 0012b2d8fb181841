"""The work that this framework's users have it do, as measurable cases.

Five kinds of program, each through the public entry points:

frame     one simulation advanced by a block of ETD1 steps, then observed: the free energy
          of the state and its real-space field. `restart` uploads the initial field first
          (a run from its initial condition); otherwise the simulation goes on from where
          the last block left it, as a long run does.
snapshot  one simulation restarted, advanced a little and observed in full: field, mu, the
          coarse-grained field, the nonlinear part of mu, F, mean mu and mean density.
cells     phase-diagram relaxations: a batch of small crystal cells, each with its own box
          scale and mean density, stepped together by one relaxation block, with the
          rollback snapshot before it and the free energies after it.
sweep     a phase-diagram sweep's block: plans of three box sizes, crystal and liquid starts,
          stepped together, F / mu / mean of every point, and every point's field.
extv      the log model with an external potential and the re-optimised linear shift.

The FP64 form's fields come back as it gives them. The FP32-mixed form computes fields in
single precision, and a program that runs it keeps its frames in single precision too.
"""
import math

import numpy as np
import torch

from pfc_models_b200 import _lib, logpfc, logpfc_extv, stdpfc, tune
from pfc_models_b200.simulation import Batch

A_CELL, H_CELL = 4 * math.pi / math.sqrt(3), 4 * math.pi   # one rectangular cell of the lattice
Q = math.sqrt(3) / 2                                       # one-mode wavenumber along x

# the models' parameter sets in the examples and workloads
STD = dict(Gamma=1.0, beta=1.0, q0=1.0, g=0.0, dt=0.5)
LOG = dict(Gamma=1.0, beta=0.5, q0=1.0, epsilon=-0.9, g=-2.0, dt=0.1)

SITE_STEPS = 8192 * 8192 * 50   # of the largest listed frame


def listed():
    return [
        # one relaxation block (stepT = 100 at dt = 0.1) of one phase-diagram cell
        dict(name="cell_28x24_log_fp64", kind="frame", model="log", precision="fp64", nx=28, ny=24, steps=1000,
             restart=False),
        # the same block for every point of a q00 scan of 12 densities
        dict(name="cells_28x24_log_fp64_x252", kind="cells", nx=28, ny=24, count=252, steps=1000),
        # the reference's own loop: one TimeStep, one look at the field
        dict(name="one_step_256_std_fp64", kind="frame", model="std", precision="fp64", nx=256, ny=256, steps=1,
             restart=False),
        # the 256^2 configuration between two records, from its initial field
        dict(name="frame_256_std_fp64", kind="frame", model="std", precision="fp64", nx=256, ny=256, steps=100,
             restart=True),
        # the 1024^2 logPFC configuration
        dict(name="frame_1024_log_fp32", kind="frame", model="log", precision="fp32", nx=1024, ny=1024, steps=100,
             restart=False),
        # the 2048^2 polycrystal in both precision forms
        dict(name="frame_2048_std_fp32", kind="frame", model="std", precision="fp32", nx=2048, ny=2048, steps=128,
             restart=False),
        dict(name="frame_2048_std_fp64", kind="frame", model="std", precision="fp64", nx=2048, ny=2048, steps=32,
             restart=False),
        # the 8192^2 solidification between two free-energy records
        dict(name="frame_8192_std_fp32", kind="frame", model="std", precision="fp32", nx=8192, ny=8192, steps=50,
             restart=False),
        # an eighth or so of the 512-point sweep
        dict(name="sweep_72_fp32", kind="sweep", precision="fp32", count=72, steps=200),
        # 16 x 28 cells tiled to sides with the factor 7 twice: transforms planned at run time
        dict(name="frame_896x1568_std_fp64", kind="frame", model="std", precision="fp64", nx=896, ny=1568, steps=32,
             restart=False),
        # every observable of a freshly uploaded field on sides with one odd factor
        dict(name="snapshot_1536_log_fp32", kind="snapshot", model="log", precision="fp32", nx=1536, ny=1536, steps=8),
        # the external-potential model's smoke configuration (sides with the factor 11)
        dict(name="extv_264_log_fp64", kind="extv", nx=264, ny=264, steps=100),
    ]


# ------------------------------------------------------------------ drawn cases
def _smooth(limit, primes=(2, 3, 5, 7, 11, 13)):
    out = {1}
    for p in primes:
        grown = set(out)
        for v in out:
            while v * p <= limit:
                v *= p
                grown.add(v)
        out = grown
    return sorted(out)


# plans refuse some long sides with the factors 11 and 13
_SIDES = [v for v in _smooth(2048) if v >= 16 and (v <= 1024 or v in set(_smooth(2048, (2, 3, 5, 7))))]


def _side(rng, low, high, even):
    """A side the plans take, spread over the logarithm of [low, high]: half of the time a
    power of two, else any length with factors up to 13."""
    want = math.exp(rng.uniform(math.log(low), math.log(high)))
    if rng.random() < 0.5:
        return min(max(2 ** round(math.log2(want)), low), high)
    ok = [v for v in _SIDES if low <= v <= high and (not even or v % 2 == 0)]
    return min(ok, key=lambda v: abs(math.log(v / want)))


def draw(rng):
    kind = rng.choice(["frame"] * 6 + ["snapshot", "cells", "sweep", "extv"])
    if kind == "cells":
        nx, ny = rng.choice([(28, 24), (14, 24), (16, 28), (32, 56), (20, 36), (48, 20), (30, 22)])
        return dict(kind=kind, nx=nx, ny=ny, count=rng.randint(2, 252), steps=rng.randint(20, 1000))
    if kind == "sweep":
        return dict(kind=kind, precision=rng.choice(["fp32", "fp64"]), count=rng.randint(3, 72),
                    steps=rng.randint(16, 200))
    if kind == "extv":
        nx, ny = _side(rng, 32, 512, True), _side(rng, 32, 512, False)
        return dict(kind=kind, nx=nx, ny=ny, steps=rng.randint(5, 100))
    nx, ny = _side(rng, 32, 2048, True), _side(rng, 32, 2048, False)
    if kind == "frame" and rng.random() < 0.15:
        nx, ny = rng.choice([(4096, 4096), (4096, 2048), (2048, 4096), (8192, 4096), (8192, 8192)])
    case = dict(kind=kind, model=rng.choice(["std", "log"]), precision=rng.choice(["fp32", "fp64"]), nx=nx, ny=ny)
    # at most an eighth of the largest listed frame's site-steps: run-time transforms in the
    # FP64 form cost about five times its time a site
    most = min(1000 if case["precision"] == "fp64" else 128, max(1, SITE_STEPS // (8 * nx * ny)))
    case["steps"] = int(round(math.exp(rng.uniform(0.0, math.log(most))))) if kind == "frame" else rng.randint(1, 8)
    if kind == "frame":
        case["restart"] = rng.random() < 0.3
    return case


# ------------------------------------------------------------------ inputs
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) % (1 << 62))


def _one_mode(X, Y, A, scale=1.0):
    q = Q * scale
    return A * (torch.cos(q * X) * torch.cos(q * Y / math.sqrt(3)) - 0.5 * torch.cos(2 * q * Y / math.sqrt(3)))


def _grid(nx, ny, lx, ly):
    x = torch.arange(nx, dtype=torch.float64, device="cuda") * (lx / nx)
    y = torch.arange(ny, dtype=torch.float64, device="cuda") * (ly / ny)
    return x[None, :], y[:, None]


def _box(case):
    if case["model"] == "log":   # whole cells, about pi / 4 a site as in the 1024^2 configuration
        return (max(1, round(case["nx"] * 108 / 1024)) * A_CELL, max(1, round(case["ny"] * 62 / 1024)) * H_CELL)
    return case["nx"] * math.pi / 4, case["ny"] * math.pi / 4


def _polycrystal(case, seed):
    """Noisy liquid with circular crystal grains of radius 12 sites at random places and angles."""
    nx, ny = case["nx"], case["ny"]
    lx, ly = _box(case)
    log = case["model"] == "log"
    mean, A, radius = (0.55, 0.2, 12 * lx / nx) if log else (-0.28, 0.5, 12 * math.pi / 4)
    gen = _generator(seed)
    f = mean + 0.01 * (2 * torch.rand((ny, nx), generator=gen, dtype=torch.float64, device="cuda") - 1)
    host = np.random.default_rng(int(seed) % (1 << 62))
    if min(nx, ny) >= 64:
        w = 14
        dx, dy = lx / nx, ly / ny
        for _ in range(max(1, min(256, nx * ny // 65536))):
            ix, iy = host.integers(0, nx), host.integers(0, ny)
            th = host.uniform(0, math.pi / 3)
            at = torch.arange(-w, w + 1, device="cuda")
            px, py = (at * dx)[None, :].double(), (at * dy)[:, None].double()
            X, Y = math.cos(th) * px + math.sin(th) * py, math.cos(th) * py - math.sin(th) * px
            jx, jy = ((at + int(ix)) % nx)[None, :], ((at + int(iy)) % ny)[:, None]
            f[jy, jx] = torch.where(px * px + py * py < radius * radius, mean + _one_mode(X, Y, A), f[jy, jx])
    return f


def _cell_points(case, seed):
    """(mean density, box scale) of each relaxation and its crystal ansatz on the 2 x 1 (or
    the nearest whole) cell."""
    host = np.random.default_rng(int(seed) % (1 << 62))
    count = case.get("count", 1)
    mean = host.uniform(0.50, 0.62, count)
    q00 = host.uniform(0.97, 1.03, count)
    mx, my = max(1, round(case["nx"] / 14)), max(1, round(case["ny"] / 24))
    gen = _generator(seed)
    fields = []
    for m, q in zip(mean, q00):
        lx, ly = mx * A_CELL / q, my * H_CELL / q
        X, Y = _grid(case["nx"], case["ny"], lx, ly)
        f = m * (1 + _one_mode(X, Y, 0.3, q))
        f = f * (1 + 1e-3 * torch.randn(f.shape, generator=gen, dtype=torch.float64, device="cuda"))
        fields.append((lx, ly, f))
    return fields


_SWEEP_BOXES = ((128, 14, 8), (256, 28, 16), (512, 56, 32))


def _sweep_points(case, seed):
    host = np.random.default_rng(int(seed) % (1 << 62))
    gen = _generator(seed)
    out = []
    for i in range(case["count"]):
        n, mx, my = _SWEEP_BOXES[i % 3]
        # densities from the limit of stability of the liquid on, where the tangent points lie
        r = host.uniform(-0.6, -0.05)
        psi = -math.sqrt(-r / 3) * host.uniform(1.0, 1.3)
        lx, ly = mx * A_CELL, my * H_CELL
        # noise in the crystals too: a perfect one would break its symmetry by rounding alone
        f = psi + 0.01 * (2 * torch.rand((n, n), generator=gen, dtype=torch.float64, device="cuda") - 1)
        if (i // 3) % 2 == 0:
            X, Y = _grid(n, n, lx, ly)
            f = f + _one_mode(X, Y, 0.5)
        out.append((n, r, lx, ly, f))
    return out


def _extv_input(case, seed):
    """Crystal with noise, and a Gaussian dipole potential."""
    nx, ny = case["nx"], case["ny"]
    lx, ly = max(1, round(nx / 22)) * A_CELL, max(1, round(ny / 22 * A_CELL / H_CELL)) * H_CELL
    X, Y = _grid(nx, ny, lx, ly)
    gen = _generator(seed)
    f = 0.55 * (1 + _one_mode(X, Y, 0.4)) + 1e-3 * (torch.rand((ny, nx), generator=gen, dtype=torch.float64,
                                                                device="cuda") - 0.5)
    return lx, ly, f, (0.02, (0.3 * lx, 0.4 * ly), (0.7 * lx, 0.6 * ly), 3.0)


# ------------------------------------------------------------------ what a program has in hand
def _simulation(case, lx, ly):
    if case["model"] == "log":
        return logpfc.BuildB200_Simulation(logpfc.BuildLogPFCModelParameters(**LOG),
                                           logpfc.Build2DGeometry(case["nx"], case["ny"], lx, ly),
                                           precision=case["precision"])
    return stdpfc.BuildB200_Simulation(stdpfc.BuildStdPFCModelParameters(epsilon=-0.25, **STD),
                                       stdpfc.Build2DGeometry(case["nx"], case["ny"], lx, ly),
                                       precision=case["precision"])


def _density(sim):
    return sim.State.phi if sim.model == "log" else sim.State.n


def _small_cell(case):
    return case["model"] == "log" and case["nx"] * case["ny"] <= 2048


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("frame", "snapshot"):
        if _small_cell(case):
            lx, ly, field = _cell_points(case, seed)[0]
        else:
            (lx, ly), field = _box(case), _polycrystal(case, seed)
        sim = _simulation(case, lx, ly)
        _density(sim)[...] = field
        return dict(case=case, sim=sim, field=field)
    if kind == "cells":
        sims = []
        for lx, ly, field in _cell_points(case, seed):
            sim = _simulation(dict(case, model="log", precision="fp64"), lx, ly)
            sim.State.phi[...] = field
            sims.append(sim)
        return dict(case=case, sims=sims, batch=Batch(sims))
    if kind == "sweep":
        sims = []
        code = _lib.FP32_MIXED if case["precision"] == "fp32" else _lib.FP64_PLAIN
        for n, r, lx, ly, field in _sweep_points(case, seed):
            prm = stdpfc.BuildStdPFCModelParameters(epsilon=r, **STD)
            kernels = tune.lookup(n, n, code, _lib.MODEL_STD, batched=True) or "auto"
            sim = stdpfc.BuildB200_Simulation(prm, stdpfc.Build2DGeometry(n, n, lx, ly), precision=case["precision"],
                                              kernels=kernels)
            sim.State.n[...] = field
            sims.append(sim)
        return dict(case=case, sims=sims, batch=Batch(sims))
    lx, ly, field, dipole = _extv_input(case, seed)
    prm = logpfc_extv.BuildLogPFCModel_withVacancyForce_Parameters(meanDensity=0.55, **LOG)
    sim = logpfc_extv.BuildB200_Simulation(prm, logpfc_extv.BuildGeometry(case["nx"], case["ny"], lx, ly))
    sim.State.phi[...] = field
    sim._externalV.SetGaussianDipolePotential(*dipole)
    return dict(case=case, sim=sim, field=field)


# ------------------------------------------------------------------ one pass
def _kept(case, t):
    return t.float() if case.get("precision") == "fp32" else t


def _number(case, v):
    return np.float32(v) if case.get("precision") == "fp32" else np.float64(v)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("cells", "sweep"):
        sims, batch = state["sims"], state["batch"]
        if kind == "cells":
            before = [sim.plan.get_state() for sim in sims]
            batch.step(case["steps"])
            return dict(before=torch.stack(before), table=batch.reduce(),
                        after=torch.stack([sim.State.phi.torch() for sim in sims]))
        batch.step(case["steps"])
        table = batch.reduce()
        return dict(table=table.astype(np.float32) if case["precision"] == "fp32" else table,
                    fields=torch.cat([_kept(case, sim.State.n.torch()).flatten() for sim in sims]))
    sim = state["sim"]
    if kind == "snapshot" or case.get("restart"):
        _density(sim)[...] = state["field"]
    if case["steps"] == 1:
        sim.TimeStep()
    else:
        sim.TimeSteps(case["steps"])
    if kind == "snapshot":
        F, mu, mean = sim.Reduce()
        local = sim.Get_local_phi() if sim.model == "log" else sim.Get_local_n()
        return dict(field=_kept(case, _density(sim).torch()), mu=_kept(case, sim.State.mu.torch()),
                    nonlin_mu=_kept(case, sim.State.nonlin_mu.torch()),
                    local=local.astype(np.float32) if case["precision"] == "fp32" else local,
                    F=_number(case, F), mean_mu=_number(case, mu), mean=_number(case, mean))
    if case["steps"] == 1:
        return dict(field=_kept(case, _density(sim).torch()))
    return dict(F=_number(case, sim.CalculateFreeEnergy()), field=_kept(case, _density(sim).torch()))


# ------------------------------------------------------------------ the work of a pass
def _grids(case):
    if case["kind"] == "sweep":
        return [(_SWEEP_BOXES[i % 3][0],) * 2 for i in range(case["count"])]
    return [(case["nx"], case["ny"])] * case.get("count", 1)


def work(case):
    """A step takes the spectral state and both directions of two 2-D real transforms through
    memory: six passes over a half spectrum. The small cells stay on the chip for the whole
    block and need their field in and out once. A real transform of N sites is 2.5 N log2 N."""
    elt = 4 if case.get("precision") == "fp32" else 8
    b = f = 0.0
    for nx, ny in _grids(case):
        n = nx * ny
        passes = 1 if n <= 2048 else case["steps"]
        b += 6 * elt * n * passes + 2 * 8 * n
        f += case["steps"] * n * (2 * 2.5 * math.log2(n) + 20)
        if case["kind"] == "snapshot":
            b += 4 * 8 * n
            f += n * 4 * 2.5 * math.log2(n)
    return {"bytes": b, "flops": f}


# ------------------------------------------------------------------ 64-bit values, plain torch
class _Exact:
    """The pseudo-spectral ETD1 stepper in 64 bits over a stack of equal grids."""

    def __init__(self, model, fields, lx, ly, epsilon, p, tol=2e-5):
        self.model, self.p, self.n = model, p, fields.clone()
        ny, nx = fields.shape[-2:]
        col = lambda v: torch.as_tensor(v, dtype=torch.float64, device="cuda").reshape(-1, 1, 1)  # noqa: E731
        kx = 2 * math.pi * torch.arange(nx // 2 + 1, dtype=torch.float64, device="cuda")[None, None, :] / col(lx)
        iy = torch.arange(ny, dtype=torch.float64, device="cuda")
        iy = torch.where(iy <= (ny - 1) // 2, iy, iy - ny)
        ky = 2 * math.pi * iy[None, :, None] / col(ly)
        self.lap, self.eps, self.shape, self.tol = -(kx * kx + ky * ky), col(epsilon), (ny, nx), tol
        self.lin_mu = p["beta"] * (p["q0"] ** 2 + self.lap) ** 2 + self.eps
        self.shift(0.0)
        self.nhat = self.prev = None

    def shift(self, M):
        p = self.p
        L = p["Gamma"] * self.lap * (self.lin_mu + M)
        z = L * p["dt"]
        self.A1 = torch.expm1(z)
        small = z.abs() <= self.tol
        self.B = torch.where(small, p["dt"] * (1 + z / 2 + z * z / 6), self.A1 / torch.where(small, torch.ones_like(L), L))

    def nonlin(self, n):
        r = self.p["g"] * n * n + n * n * n
        return r + torch.log(n) if self.model == "log" else r

    def step(self, M=None, force=None, min_phi=None):
        n = self.n
        N = self.nonlin(n)
        if M is not None:
            N = torch.where(n > min_phi, torch.log(n), math.log(min_phi)) + self.p["g"] * n * n + n * n * n - M * n
        self.prev = n
        h, q = torch.fft.rfft2(n), torch.fft.rfft2(N)
        q *= self.p["Gamma"] * self.lap
        if force is not None:
            q += self.lap * force
        h += self.A1 * h + self.B * q
        self.n = torch.fft.irfft2(h, s=self.shape)

    def energy(self):
        p, n = self.p, self.n
        lin = torch.fft.irfft2(0.5 * p["beta"] * (p["q0"] ** 2 + self.lap) ** 2 * torch.fft.rfft2(n), s=self.shape)
        f = 0.5 * self.eps * n * n + p["g"] / 3 * n ** 3 + 0.25 * n ** 4
        if self.model == "log":
            f = f + n * torch.log(n)
        return (n * lin + f).mean(dim=(-2, -1))

    def mean_mu(self):
        p = self.p
        lin = (p["beta"] * p["q0"] ** 4 + self.eps).reshape(-1)
        return lin * self.n.mean(dim=(-2, -1)) + self.nonlin(self.n).mean(dim=(-2, -1))

    def table(self):
        return torch.stack([self.energy(), self.mean_mu(), self.n.mean(dim=(-2, -1))], dim=1)


def exact(case, seed):
    kind, steps = case["kind"], case["steps"]
    if kind == "cells":
        pts = _cell_points(case, seed)
        before = torch.stack([f for _, _, f in pts])
        e = _Exact("log", before, [p[0] for p in pts], [p[1] for p in pts], LOG["epsilon"], LOG)
        for _ in range(steps):
            e.step()
        return dict(before=before, table=e.table().cpu().numpy(), after=e.n)
    if kind == "sweep":
        pts = _sweep_points(case, seed)
        table, fields = [None] * len(pts), [None] * len(pts)
        for n in sorted({p[0] for p in pts}):
            at = [i for i, p in enumerate(pts) if p[0] == n]
            e = _Exact("std", torch.stack([pts[i][4] for i in at]), [pts[i][2] for i in at], [pts[i][3] for i in at],
                       [pts[i][1] for i in at], STD)
            for _ in range(steps):
                e.step()
            for k, row in zip(at, e.table()):
                table[k] = row
            for k, f in zip(at, e.n):
                fields[k] = f.flatten()
        return dict(table=torch.stack(table).cpu().numpy(), fields=torch.cat(fields))
    if kind == "extv":
        lx, ly, field, (V0, (x0, y0), (x1, y1), s) = _extv_input(case, seed)
        e = _Exact("log", field[None], lx, ly, LOG["epsilon"], LOG, tol=1e-8)
        X, Y = _grid(case["nx"], case["ny"], lx, ly)
        V = V0 * (torch.exp(-((X - x0) ** 2 + (Y - y0) ** 2) / (2 * s * s))
                  - torch.exp(-((X - x1) ** 2 + (Y - y1) ** 2) / (2 * s * s)))
        force = torch.fft.rfft2(V)[None]
        bounds, M = None, 0.0
        for _ in range(steps):
            lo, hi = float(e.n.min()), float(e.n.max())
            if bounds is None or (bounds[0] - lo) / bounds[0] > 0.1 or (hi - bounds[1]) / bounds[1] > 0.1:
                lo = lo if lo > 0 else 1e-6
                N = lambda x: LOG["g"] * x ** 2 + x ** 3 + math.log(x)  # noqa: E731
                M, bounds = (N(hi) - N(lo)) / (hi - lo), (lo, hi)
                e.shift(M)
            e.step(M, force, 1e-6)
        return dict(F=np.float64(e.energy().item()), field=e.n[0])
    if _small_cell(case):
        lx, ly, field = _cell_points(case, seed)[0]
    else:
        (lx, ly), field = _box(case), _polycrystal(case, seed)
    p = LOG if case["model"] == "log" else STD
    e = _Exact(case["model"], field[None], lx, ly, LOG["epsilon"] if case["model"] == "log" else -0.25, p)
    for _ in range(steps):
        e.step()
    if kind == "snapshot":
        prev = e.prev
        N = e.nonlin(prev)
        mu = torch.fft.irfft2(e.lin_mu * torch.fft.rfft2(prev) + torch.fft.rfft2(N), s=e.shape)
        local = torch.fft.irfft2(torch.exp(0.5 * e.lap * (2 * math.pi) ** 2) * torch.fft.rfft2(prev), s=e.shape)
        F, mean_mu, mean = e.table()[0].cpu().numpy()
        return dict(field=e.n[0], mu=mu[0], nonlin_mu=N[0], local=local[0].cpu().numpy(), F=F, mean_mu=mean_mu, mean=mean)
    if steps == 1:
        return dict(field=e.n[0])
    return dict(F=np.float64(e.energy().item()), field=e.n[0])
