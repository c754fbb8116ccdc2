"""The work a user of cpic_gb300 has it do, as measurable cases.

Six kinds of work, each through the public entry points as a program calls
them:

  poisson   the Poisson solve on the caller's own device buffers;
  sim       a prepared simulation advanced by some steps, then the read-out
            a program writes at an output interval (charge density, E, and
            on small runs the particles);
  loop      the same, step by step, with the field energy read after every
            step (the driver loop of a diagnostic run);
  job       a whole run from host arrays: set-up, upload, steps, read-out,
            download of the particles, tear-down;
  ensemble  independent runs of different sizes stepped together;
  adjoint   the field energy after a run and its gradient with respect to
            every initial position and velocity, through torch.autograd.

Units are the repository's (e0 = 1, electron q/m = -1, plasma frequency 1);
cells are square.  The mixed form stores and computes in 32 bits, and its
results are kept as such; the FP64 form's are kept in 64 bits.
"""
import ctypes
import gc
import math

import numpy as np
import torch

import cpic_gb300
from cpic_gb300 import _lib
from cpic_gb300 import autograd

L0 = 2.0 * math.pi
DT = 0.05


def listed():
    return [
        # the smallest call: one solve on a small grid, in a caller's own
        # loop where nothing may be allocated; bound by latency
        dict(name="poisson_64", kind="poisson", nx=64, ny=64),
        # the same at the largest grid that entry point takes
        dict(name="poisson_512", kind="poisson", nx=512, ny=512),
        # the reference's CPU-runnable size: 10,240 electrons on 64 x 64 with
        # the field energy read every step; launches and round trips count
        dict(name="loop_64_fp64", kind="loop", precision="fp64", nx=64, ny=64, n=10240, species=1,
             bz=0.0, steps=20, ids=True, particles=True),
        # two species in a magnetic field at the plain form's working size
        dict(name="sim_512_fp64_bz", kind="sim", precision="fp64", nx=512, ny=512, n=4194304,
             species=2, bz=0.5, steps=10, ids=True, particles=False),
        # a ragged grid (mixed-radix solve, 2-cell tiles) in the plain form
        dict(name="sim_250x150_fp64", kind="sim", precision="fp64", nx=250, ny=150, n=600011,
             species=1, bz=0.0, steps=10, ids=True, particles=True),
        # the headline size: 2048 x 2048 with 100 electrons per cell, written
        # out every 50 steps
        dict(name="sim_2048_mixed", kind="sim", precision="mixed", nx=2048, ny=2048, n=419430400,
             species=1, bz=0.0, steps=50, ids=False, particles=False),
        # a ragged grid of ordinary size in the mixed form
        dict(name="sim_600x400_mixed", kind="sim", precision="mixed", nx=600, ny=400, n=15360000,
             species=1, bz=0.0, steps=20, ids=False, particles=False),
        # a small two-species mixed run with particle ids, as a parameter
        # scan runs many of
        dict(name="loop_128_mixed_bz", kind="loop", precision="mixed", nx=128, ny=128, n=262144,
             species=2, bz=0.5, steps=20, ids=True, particles=True),
        # a whole mixed run from host arrays and back
        dict(name="job_256_mixed", kind="job", precision="mixed", nx=256, ny=256, n=2097152,
             species=1, bz=0.0, steps=100, ids=True, particles=True),
        # a batch of independent runs
        dict(name="ensemble_24", kind="ensemble", runs=24, smax=256, steps=50),
        # gradients: the repository's adjoint workload, FP64
        dict(name="adjoint_128_fp64", kind="adjoint", precision="fp64", nx=128, ny=128, n=1048576,
             bz=0.0, steps=200, keep=20),
        # a smaller gradient in 32 bits
        dict(name="adjoint_64_mixed", kind="adjoint", precision="mixed", nx=64, ny=64, n=262144,
             bz=0.0, steps=50, keep=10),
    ]


def _logi(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _side(rng, lo, hi):
    """A grid side: usually a power of two or a multiple of 8, sometimes odd
    or barely even."""
    v = rng.random()
    if v < 0.4:
        return 1 << rng.randint(int(math.ceil(math.log2(lo))), int(math.log2(hi)))
    s = _logi(rng, lo, hi)
    if v < 0.75:
        return max(8, s // 8 * 8)
    if v < 0.9:
        return max(4, s // 2 * 2)
    return min(s, 255) | 1


def draw(rng):
    kind = rng.choice(["poisson", "loop", "sim", "sim", "sim", "job", "ensemble", "adjoint"])
    if kind == "poisson":
        return dict(kind=kind, nx=1 << rng.randint(2, 9), ny=1 << rng.randint(2, 9))
    if kind == "ensemble":
        return dict(kind=kind, runs=rng.randint(4, 28), smax=rng.choice([64, 128, 256]),
                    steps=rng.randint(10, 60))
    precision = rng.choice(["fp64", "mixed"])
    if kind == "adjoint":
        steps = _logi(rng, 10, 100)
        nx, ny = 1 << rng.randint(4, 8), 1 << rng.randint(4, 8)
        return dict(kind=kind, precision=precision, nx=nx, ny=ny,
                    n=min(600000, nx * ny * rng.randint(4, 64) + rng.randint(0, 999)),
                    bz=rng.choice([0.0, 0.3]), steps=steps, keep=rng.randint(4, 20))
    small = kind == "loop"
    nx, ny = _side(rng, 16, 256 if small else 1024), _side(rng, 16, 256 if small else 1024)
    ppc = math.exp(rng.uniform(math.log(2.0), math.log(128.0)))
    top = 1 << 20 if small else 1 << 22 if kind == "job" else 1 << 25 if precision == "mixed" else 1 << 23
    n = max(64, min(top, int(nx * ny * ppc)))
    species = rng.choice([1, 1, 2])
    return dict(kind=kind, precision=precision, nx=nx, ny=ny, n=n, species=species,
                bz=rng.choice([0.0, 0.5]), steps=rng.randint(5, 40),
                ids=kind == "job" or precision == "fp64" or rng.random() < 0.5,
                particles=kind == "job")


# ------------------------------------------------------------------ inputs

def _gen(seed, salt):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed * 1000003 + salt)
    return g


def _beams(g, n, L, Ly, v0, vth, amp):
    """Two counter-streaming beams with a sinusoidal density perturbation."""
    kw = dict(device="cuda", dtype=torch.float64, generator=g)
    x = torch.rand(n, **kw) * L
    x = torch.remainder(x + amp * torch.sin(2 * math.pi / L * x), L)
    x[x >= L] = 0.0
    y = torch.rand(n, **kw) * Ly
    y[y >= Ly] = 0.0
    ux = torch.randn(n, **kw) * vth
    ux[:n // 2] += v0
    ux[n // 2:] -= v0
    uy = torch.randn(n, **kw) * vth
    return x, y, ux, uy


def _thermal(g, n, L, Ly, vth):
    kw = dict(device="cuda", dtype=torch.float64, generator=g)
    x, y = torch.rand(n, **kw) * L, torch.rand(n, **kw) * Ly
    x[x >= L] = 0.0
    y[y >= Ly] = 0.0
    return x, y, torch.randn(n, **kw) * vth, torch.randn(n, **kw) * vth


def _species(case, seed, salt=0):
    """[(q, m, (x, y, ux, uy) on the GPU)] of a case."""
    nx, ny, n = case["nx"], case["ny"], case["n"]
    L, Ly = L0, L0 * ny / nx
    q = -L * Ly / n
    g = _gen(seed, 17 + salt)
    if case.get("species", 1) == 1:
        return [(q, -q, _beams(g, n, L, Ly, case.get("v0", 0.2), 0.01, case.get("amp", 0.01)))]
    return [(q, -q, _thermal(g, n, L, Ly, 0.05)), (-q, -100.0 * q, _thermal(g, n, L, Ly, 0.005))]


def _host(case, seed, salt=0):
    """The same as host arrays, which the entry points take."""
    out = [(q, m, [t.cpu().numpy() for t in a]) for q, m, a in _species(case, seed, salt)]
    torch.cuda.empty_cache()
    return out


def _precision(case):
    return _lib.FP64 if case.get("precision") == "fp64" else _lib.MIXED


def _context(case, species):
    L = L0
    ctx = cpic_gb300.Context(case["nx"], case["ny"], L, L * case["ny"] / case["nx"], DT, 1.0,
                             (0.0, 0.0, case.get("bz", 0.0)), precision=_precision(case),
                             track_ids=case.get("ids", True))
    for q, m, a in species:
        ctx.add_species(q, m, *a)
    return ctx


def _members(case, seed):
    """The runs of an ensemble: grids from {32, 64, 128, 256}, 8 to 128
    electrons per cell, beams of 0.1 to 0.4.  Sizes do not depend on the
    seed: they are the batch a program has planned."""
    rng = np.random.default_rng(77 + case["runs"])
    out = []
    for i in range(case["runs"]):
        side = int(rng.choice([s for s in (32, 64, 128, 256) if s <= case["smax"]]))
        ppc = int(rng.integers(8, 129))
        out.append(dict(nx=side, ny=side, n=side * side * ppc, precision="mixed", species=1, bz=0.0,
                        ids=False, steps=case["steps"], v0=float(rng.uniform(0.1, 0.4)),
                        amp=float(rng.uniform(0.001, 0.05))))
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind == "poisson":
        rho = torch.randn(case["ny"], case["nx"], device="cuda", dtype=torch.float64,
                          generator=_gen(seed, 3))
        return dict(case=case, rho=rho, phi=torch.empty_like(rho), lib=cpic_gb300.load())
    if kind in ("sim", "loop"):
        ctx = _context(case, _host(case, seed))
        gc.collect()
        ctx.pre_step()
        return dict(case=case, ctx=ctx)
    if kind == "job":
        return dict(case=case, species=_host(case, seed))
    if kind == "ensemble":
        runs = []
        for i, m in enumerate(_members(case, seed)):
            ctx = _context(m, _host(m, seed, 100 * i))
            ctx.pre_step()
            runs.append(ctx)
        return dict(case=case, runs=runs, ens=_lib.Ensemble(runs))
    if kind == "adjoint":
        (q, m, a), = _species(case, seed)
        L = L0
        adj = _lib.Adjoint(case["nx"], case["ny"], L, L * case["ny"] / case["nx"], DT, 1.0, q, m,
                                 case["n"], case["steps"], case["keep"], Bz=case["bz"],
                                 precision=_precision(case))
        return dict(case=case, adj=adj, state=[t.requires_grad_() for t in a])
    raise ValueError(kind)


# --------------------------------------------------------------- one pass

def _keep(case, a):
    """A result as the program keeps it: 64 bits from the FP64 form, the
    mixed form's 32."""
    a = torch.as_tensor(np.asarray(a)) if not isinstance(a, torch.Tensor) else a
    return a if case.get("precision") == "fp64" else a.float()


def _readout(case, ctx):
    ex, ey = ctx.E()
    out = dict(rho=_keep(case, ctx.rho()), ex=_keep(case, ex), ey=_keep(case, ey))
    if case["particles"]:
        out["particles"] = [[_keep(case, a) for a in ctx.particles(s)]
                            for s in range(case["species"])]
    return out


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "poisson":
        r = state["lib"].cpic_poisson_noalloc(
            ctypes.c_void_p(state["rho"].data_ptr()), ctypes.c_void_p(state["phi"].data_ptr()),
            case["nx"], case["ny"], ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if r != 0:
            raise RuntimeError("cpic_poisson_noalloc: %d" % r)
        return state["phi"]
    if kind == "sim":
        state["ctx"].run(case["steps"])
        return _readout(case, state["ctx"])
    if kind == "loop":
        ctx, we = state["ctx"], []
        for _ in range(case["steps"]):
            ctx.step()
            we.append(ctx.field_energy())
        return dict(_readout(case, ctx), we=_keep(case, we))
    if kind == "job":
        ctx = _context(case, state["species"])
        ctx.pre_step()
        ctx.run(case["steps"])
        out = _readout(case, ctx)
        ctx.close()
        return out
    if kind == "ensemble":
        state["ens"].run(case["steps"])
        return dict(rho=[_keep(case, c.rho()) for c in state["runs"]],
                    we=_keep(case, [c.field_energy() for c in state["runs"]]))
    loss = autograd.field_energy(state["adj"], *state["state"])
    grads = torch.autograd.grad(loss, state["state"])
    return dict(loss=_keep(case, loss.detach()), grads=[_keep(case, g) for g in grads])


# ------------------------------------------------------------------- work

def work(case):
    kind = case["kind"]
    if kind == "ensemble":
        each = [work(dict(m, kind="sim")) for m in _members(case, 0)]
        return {k: sum(w[k] for w in each) for k in ("bytes", "flops")}
    ng = case["nx"] * case["ny"]
    fft = 5.0 * ng * math.log2(ng)               # two real transforms of the grid
    if kind == "poisson":
        return {"bytes": 16.0 * ng, "flops": fft}
    t = 8 if case["precision"] == "fp64" else 4
    if kind == "adjoint":
        # forward: x, y, ux, uy read and written; backward: the same steps
        # again, keeping positions, then positions read and the four
        # adjoints read and written
        n, s = case["n"], case["steps"]
        return {"bytes": s * (28.0 * t * n + 3 * (8 + 3 * t) * ng), "flops": s * (2 * 66.0 + 90.0) * n
                + 3 * s * fft}
    n = case["n"] * case["species"]
    per, grid = (64.0, 48.0) if t == 8 else (40.0, 40.0)
    extra = 64.0 * n if kind == "job" else 32.0 * n if case.get("particles") else 0.0
    s = case["steps"]
    return {"bytes": s * (per * n + grid * ng) + extra + 24.0 * ng, "flops": s * (66.0 * n + fft)}


# ------------------------------------------------- 64 bits, plain torch

def _cic(x, y, nx, ny, dx):
    gx, gy = x / dx, y / dx
    cx, cy = torch.floor(gx).detach(), torch.floor(gy).detach()
    fx, fy = gx - cx, gy - cy
    ix, iy = cx.long() % nx, cy.long() % ny
    ix1, iy1 = (ix + 1) % nx, (iy + 1) % ny
    idx = [iy * nx + ix, iy * nx + ix1, iy1 * nx + ix, iy1 * nx + ix1]
    return idx, [(1 - fx) * (1 - fy), fx * (1 - fy), (1 - fx) * fy, fx * fy]


def _green(nx, ny, dev):
    kx = torch.arange(nx // 2 + 1, dtype=torch.float64, device=dev)
    ky = torch.arange(ny, dtype=torch.float64, device=dev)
    G = 2.0 * (torch.cos(2 * math.pi * kx / nx)[None, :] + torch.cos(2 * math.pi * ky / ny)[:, None]) - 4.0
    G[0, 0] = 1.0
    G = 1.0 / G
    G[0, 0] = 0.0
    return G


class _Plain:
    """The step in 64 bits."""

    def __init__(self, case, seed, salt=0):
        self.c, self.nx, self.ny = case, case["nx"], case["ny"]
        self.dx = L0 / self.nx
        self.L, self.Ly = L0, L0 * self.ny / self.nx
        self.sp = [[q, m, *a] for q, m, a in _species(case, seed, salt)]
        self.G = _green(self.nx, self.ny, "cuda")
        self.j = 0
        self.deposit()

    def deposit(self):
        rho = torch.zeros(self.nx * self.ny, dtype=torch.float64, device="cuda")
        for q, m, x, y, ux, uy in self.sp:
            idx, w = _cic(x, y, self.nx, self.ny, self.dx)
            for i, ww in zip(idx, w):
                rho = rho.index_add(0, i, ww * -q)
        self.rho = rho.reshape(self.ny, self.nx)

    def field(self):
        phi = torch.fft.irfft2(self.G * torch.fft.rfft2(self.rho), s=(self.ny, self.nx))
        self.ex = (torch.roll(phi, 1, 1) - torch.roll(phi, -1, 1)) / (2 * self.dx)
        self.ey = (torch.roll(phi, 1, 0) - torch.roll(phi, -1, 0)) / (2 * self.dx)

    def energy(self):
        return 0.5 * self.dx * self.dx * (self.ex.square().sum() + self.ey.square().sum())

    def step(self):
        self.field()
        ex, ey = self.ex.reshape(-1), self.ey.reshape(-1)
        for s in self.sp:
            q, m, x, y, ux, uy = s
            idx, w = _cic(x, y, self.nx, self.ny, self.dx)
            fx = sum(ww * ex[i] for i, ww in zip(idx, w))
            fy = sum(ww * ey[i] for i, ww in zip(idx, w))
            h = 0.5 * (DT if self.j else -DT / 2) * q / m
            t = self.c.get("bz", 0.0) * h
            b = 2 * t / (1 + t * t)
            vx, vy = ux + h * fx, uy + h * fy
            px, py = vx + vy * t, vy - vx * t
            s[4], s[5] = vx + py * b + h * fx, vy - px * b + h * fy
            if self.j:
                s[2] = torch.remainder(x + DT * s[4], self.L)
                s[3] = torch.remainder(y + DT * s[5], self.Ly)
        self.j += 1
        self.deposit()

    def readout(self):
        def rows(a):
            return torch.cat([a, a[:1]])         # the ghost row E() returns
        out = dict(rho=self.rho, ex=rows(self.ex), ey=rows(self.ey))
        if self.c["particles"]:
            out["particles"] = [list(s[2:]) for s in self.sp]
        return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "poisson":
        g = _gen(seed, 3)
        rho = torch.randn(case["ny"], case["nx"], device="cuda", dtype=torch.float64, generator=g)
        G = _green(case["nx"], case["ny"], "cuda")
        return torch.fft.irfft2(G * torch.fft.rfft2(rho), s=(case["ny"], case["nx"]))
    if kind == "ensemble":
        rho, we = [], []
        for i, m in enumerate(_members(case, seed)):
            p = _Plain(m, seed, 100 * i)
            for _ in range(case["steps"]):
                p.step()
            rho.append(p.rho)
            we.append(p.energy())
        return dict(rho=rho, we=torch.stack(we))
    if kind == "adjoint":
        if case["n"] * case["steps"] > 40_000_000:
            return None                          # too much for plain autograd
        p = _Plain(case, seed)
        s = p.sp[0]
        state = [a.requires_grad_() for a in s[2:]]
        p.deposit()
        for _ in range(case["steps"]):
            p.step()
        p.field()
        loss = p.energy()
        grads = torch.autograd.grad(loss, state)
        return dict(loss=loss.detach(), grads=list(grads))
    if case["n"] * case["species"] * case["steps"] > 2_000_000_000:
        return None                              # the headline size
    p, we = _Plain(case, seed), []
    for _ in range(case["steps"]):
        p.step()
        we.append(p.energy())
    out = p.readout()
    return dict(out, we=torch.stack(we)) if kind == "loop" else out
