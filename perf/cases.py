"""Performance cases of the per-timestep update through the package's public
entry points (tenjin_gb300.host.TenjinGPU, tenjin_gb300.adjoint.AdjointRun and
the C ABI behind them).

A case names a problem (one of the builders of tenjin_gb300.cases with its
sizes), a precision and what a program does with it:

    run        a program with its fields on the GPU: set the initial
               primitives, run the time loop for a number of steps, read the
               state back (tj_set_primitive, tj_run, tj_download_domain)
    operators  a host-driven loop in the reference's own order (main.cpp:121-191):
               getTimeStep, advance, the post-advance operators, contains_nan
    exchange   the drop-in step with the state on the host: upload, step and
               download through page-locked buffers
    adjoint    forward with checkpoints, then the gradient of a density misfit
    tangent    one directional derivative of the same run

run() returns the state by physical kind, in the working type of the precision: float64 for FP64, float32 for MIXED.
"""
import ctypes
import math

import numpy as np
import torch

from tenjin_gb300 import cases as problems
from tenjin_gb300.adjoint import AdjointRun
from tenjin_gb300.host import FP64, MIXED, TenjinGPU

PRECISION = {"fp64": FP64, "mixed": MIXED}


def listed():
    return [
        # the 2-D water/air shock-bubble problem with BVD-THINC, the workload the benchmark quotes
        dict(name="bubble_1024_mixed", do="run", problem="bubble", n=1024, grid=128, thinc=1, walls=0,
             precision="mixed", steps=40),
        # the same equations on a small odd grid, MUSCL alone, between reflecting walls
        dict(name="bubble_333_mixed_muscl", do="run", problem="bubble", n=333, grid=64, thinc=0, walls=1,
             precision="mixed", steps=40),
        # the reference-order FP64 run that accuracy and parity work compares with
        dict(name="bubble_256_fp64", do="run", problem="bubble", n=256, grid=64, thinc=1, walls=0,
             precision="fp64", steps=20),
        # a batch of independent uneven 3-D boxes sharing one dt
        dict(name="boxes_128_mixed", do="run", problem="boxes", n=128, precision="mixed", steps=30),
        # elastoplastic copper plate impact (5-wave solver, radial return, cleanUpV)
        dict(name="copper_128_mixed", do="run", problem="copper", n=128, grid=64, precision="mixed", steps=5),
        dict(name="copper_40_fp64", do="run", problem="copper", n=40, grid=16, precision="fp64", steps=10),
        # a solid against a gas: two materials through the solids path in binary32
        dict(name="solid_gas_192_mixed", do="run", problem="solid_gas", n=192, grid=64, precision="mixed", steps=8),
        # the 1-D shock tube at its reference resolution: launches and latency
        dict(name="sod_1000_fp64", do="run", problem="sod", n=1000, grid=1000, precision="fp64", steps=100),
        # the reference's loop driven operator by operator on a small grid: the smallest calls
        dict(name="operators_64_fp64", do="operators", problem="bubble", n=64, grid=32, thinc=1, walls=0,
             precision="fp64", steps=5),
        # a host code that owns the state and hands it over every step
        dict(name="exchange_1024_mixed", do="exchange", problem="bubble", n=1024, grid=128, thinc=1, walls=0,
             precision="mixed", steps=1),
        # gradients: the 2-D interface problem and the copper plate
        dict(name="adjoint_bubble_192", do="adjoint", problem="bubble", n=192, grid=64, thinc=1, walls=0,
             precision="fp64", steps=20, stride=10),
        dict(name="adjoint_copper_16", do="adjoint", problem="copper", n=16, grid=16, precision="fp64", steps=4,
             stride=2),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["bubble_mixed", "bubble_mixed", "bubble_fp64", "boxes", "copper_mixed", "copper_fp64",
                       "solid_gas", "sod", "operators", "exchange", "adjoint_bubble", "adjoint_copper", "tangent"])
    grid = rng.choice([32, 64, 128])
    if kind == "bubble_mixed":
        # until the shock reaches the bubble, after about 0.4 n steps: from there on the flow is chaotic, and runs
        # that differ in the last bit, in binary64 too, part to 1e-4 and more
        n = _log(rng, 40, 1024)
        return dict(do="run", problem="bubble", n=n, grid=grid, thinc=rng.choice([0, 1]), walls=rng.choice([0, 1]),
                    precision="mixed", steps=rng.randint(8, max(10, min(40, n // 5))))
    if kind == "bubble_fp64":
        return dict(do="run", problem="bubble", n=_log(rng, 40, 256), grid=grid, thinc=rng.choice([0, 1]),
                    walls=rng.choice([0, 1]), precision="fp64", steps=rng.randint(5, 20))
    if kind == "boxes":
        return dict(do="run", problem="boxes", n=_log(rng, 2, 128), precision="mixed", steps=rng.randint(5, 30))
    if kind == "copper_mixed":
        return dict(do="run", problem="copper", n=_log(rng, 12, 128), grid=grid, precision="mixed",
                    steps=rng.randint(2, 5))
    if kind == "copper_fp64":
        return dict(do="run", problem="copper", n=rng.randint(10, 40), grid=16, precision="fp64",
                    steps=rng.randint(4, 10))
    if kind == "solid_gas":
        return dict(do="run", problem="solid_gas", n=_log(rng, 20, 192), grid=grid, precision="mixed",
                    steps=rng.randint(2, 8))
    if kind == "sod":
        return dict(do="run", problem="sod", n=_log(rng, 50, 4000), grid=rng.choice([100, 1000]), precision="fp64",
                    steps=rng.randint(20, 100))
    if kind == "operators":
        return dict(do="operators", problem="bubble", n=_log(rng, 20, 200), grid=32, thinc=rng.choice([0, 1]),
                    walls=0, precision="fp64", steps=rng.randint(1, 5))
    if kind == "exchange":
        return dict(do="exchange", problem="bubble", n=_log(rng, 64, 1024), grid=128, thinc=1, walls=0,
                    precision="mixed", steps=1)
    if kind == "adjoint_bubble":
        return dict(do="adjoint", problem="bubble", n=_log(rng, 24, 192), grid=64, thinc=1, walls=0, precision="fp64",
                    steps=rng.randint(4, 20), stride=rng.randint(2, 10))
    if kind == "adjoint_copper":
        return dict(do="adjoint", problem="copper", n=rng.randint(6, 16), grid=16, precision="fp64",
                    steps=rng.randint(2, 4), stride=2)
    return dict(do="tangent", problem="copper", n=rng.randint(8, 24), grid=16, precision="fp64", steps=4)


# ---------------------------------------------------------------------------
# Inputs.
# ---------------------------------------------------------------------------
def _problem(case, seed):
    n, kind = case["n"], case["problem"]
    if kind == "bubble":
        # gradients need a base state that is nowhere exactly uniform (the limiter is not differentiable there)
        bg = 1e-3 if case["do"] in ("adjoint", "tangent") else 0.0
        c = problems.shock_bubble_2d(n=n, seed=seed, max_grid_size=case["grid"], thinc=case["thinc"], background=bg)
        if case["walls"]:
            c.lo_bc = [0, problems.BC_REFLECTIVE, 0]
            c.hi_bc = [problems.BC_REFLECTIVE, problems.BC_REFLECTIVE, 0]
        return c
    if kind == "boxes":
        # the boxes are the case's; the seed's are their pressure noise and, in each, a slab of compressed fluid
        # (10 to 100 MPa over the lower part of one axis) that sends a shock through the box
        c = problems.uneven_boxes_3d(nbox=n, seed=n)
        rng = np.random.Generator(np.random.PCG64(seed))
        for d in c.domains:
            axis = int(rng.integers(3))
            part = np.moveaxis(d.prim[7], axis, 0)
            d.prim[7] = problems.AMBIENT_P * (1.0 + 0.1 * rng.uniform(size=d.prim[7].shape))
            part[:int(len(part) * rng.uniform(0.2, 0.8))] += 10.0 ** rng.uniform(7.0, 8.0)
        return c
    if kind == "copper":
        return problems.copper_plate_3d(n=n, seed=seed, max_grid_size=case["grid"])
    if kind == "solid_gas":
        return problems.solid_mixture_2d(problems.EOS_WILKINS, n=n, seed=seed, max_grid_size=case["grid"])
    c = problems.sod_1d(ncells=n, max_grid_size=case["grid"])
    rng = np.random.Generator(np.random.PCG64(seed))
    x = (np.arange(n) + 0.5) / n
    for row in (2, 3, 7):  # densities and pressure: the two states, with a seeded smooth variation
        c.domains[0].prim[row, 0, 0] *= 1.0 + 0.05 * np.sin(2 * np.pi * (rng.integers(1, 4) * x + rng.uniform()))
    return c


def _groups(c, precision):
    """Component indices of the state by physical kind (AccessPattern order): the
    conservative variables, velocity, pressure, strain, and in FP64 the
    materials' own densities (alphaRho / alpha: in binary32, and in trace
    amounts, the quotient of two numbers near zero)."""
    M = c.M
    b = 3 * M + 1
    g = {"alpha": list(range(M)), "alpha_rho": list(range(M, 2 * M)), "momentum": list(range(b, b + 3)),
         "velocity": list(range(b + 3, b + 6)), "energy": [b + 6], "pressure": [b + 7]}
    if precision == "fp64":
        g["rho_k"] = list(range(2 * M, 3 * M))
    if c.solid:
        v = b + 8 + 11
        g["strain"] = list(range(v, v + 9)) + [v + 27]
        if c.plastic:
            g["strain"] += list(range(v + 28, v + 28 + M))
            g["alpha_rho_strain"] = g.pop("alpha_rho") + list(range(v + 28 + M, v + 28 + 2 * M))
    return g


def _dp(t, at=0):
    return ctypes.cast(ctypes.c_void_p(t.data_ptr() + 8 * at), ctypes.POINTER(ctypes.c_double))


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case = case
    c = s.c = _problem(case, seed)
    s.dtype = torch.float64 if case["precision"] == "fp64" else torch.float32
    s.groups = _groups(c, case["precision"])
    if case["do"] in ("adjoint", "tangent"):
        s.run = AdjointRun(c)
        s.dts = s.run.dt_schedule(case["steps"])
        s.eos = s.run.eos_array()
        s.prim = torch.from_numpy(np.ascontiguousarray(c.domains[0].prim)).cuda()
        rng = np.random.Generator(np.random.PCG64(seed + 1))
        shape = s.run.shape_state[1:]
        if case["do"] == "adjoint":
            # the weights of a linear misfit: one smooth-free random field per partial density
            s.grad = torch.zeros(s.run.shape_state, dtype=torch.float64)
            s.grad[c.M:2 * c.M] = torch.from_numpy(rng.standard_normal((c.M,) + shape))
            s.grad = s.grad.cuda()
        else:
            v = rng.standard_normal(c.domains[0].prim.shape) * np.abs(c.domains[0].prim) * 1e-3
            s.dprim = torch.from_numpy(np.ascontiguousarray(v)).cuda()
        return s
    s.sim = TenjinGPU(c, PRECISION[case["precision"]], set_initial=False)
    nc = s.sim.ncomp
    cells = [d.ncells for d in c.domains]
    if case["do"] == "exchange":
        # the host's own page-locked buffers, in the reference's layout
        d = c.domains[0]
        shape = (nc, d.n_cells[2], d.n_cells[1], d.n_cells[0])
        s.host_in = torch.empty(shape, dtype=torch.float64, pin_memory=True)
        s.host_out = torch.zeros(shape, dtype=torch.float64, pin_memory=True)
        s.sim.set_primitive(0, d.prim)
        s.sim.state(0, out=s.host_in.numpy())
        return s
    s.prim = torch.from_numpy(np.concatenate([d.prim.ravel() for d in c.domains])).cuda()
    s.out = torch.empty(nc * sum(cells), dtype=torch.float64, device="cuda")
    s.prim_at, s.out_at = [0], [0]
    for m in cells:
        s.prim_at.append(s.prim_at[-1] + c.nprim * m)
        s.out_at.append(s.out_at[-1] + nc * m)
    if len(cells) > 1:
        s.pick = {k: torch.cat([torch.arange(s.out_at[q] + g[0] * m, s.out_at[q] + (g[-1] + 1) * m, dtype=torch.int32)
                                for q, m in enumerate(cells)]).cuda() for k, g in s.groups.items()}
    return s


def _fields(s, out):
    """The state by physical kind from the downloaded planes."""
    if len(s.c.domains) > 1:
        return {k: out[i].to(s.dtype) for k, i in s.pick.items()}
    planes = out.view((-1,) + tuple(s.c.domains[0].n_cells[::-1]))
    parts = {}
    for k, g in s.groups.items():
        whole = len(g) == g[-1] - g[0] + 1
        parts[k] = (planes[g[0]:g[-1] + 1] if whole else planes[g]).to(s.dtype)
    return parts


def run(s):
    case = s.case
    if case["do"] == "adjoint":
        state = s.run.forward(s.prim, s.eos, s.dts, case["stride"])
        grad_prim, grad_eos = s.run.backward(s.grad)
        return {"state": _fields(s, state.view(-1)), "grad_prim": grad_prim, "grad_eos": grad_eos}
    if case["do"] == "tangent":
        state, dstate = s.run.tangent(s.prim, s.dprim, s.eos, None, s.dts, want_state=True)
        return {"state": _fields(s, state.view(-1)), "tangent": _fields(s, dstate.view(-1))}
    sim = s.sim
    sim._check(sim.L.tj_set_time(sim.h, 0.0, 0))
    if case["do"] == "exchange":
        sim.set_state(0, s.host_in.numpy())
        sim.step()
        return _fields(s, torch.from_numpy(sim.state(0, out=s.host_out.numpy())).view(-1))
    for q in range(len(s.c.domains)):
        sim._check(sim.L.tj_set_primitive(sim.h, q, _dp(s.prim, s.prim_at[q])))
    if case["do"] == "operators":
        dts = []
        for n in range(case["steps"]):
            dt = sim.getTimeStep() * (0.2 if n < 5 else 1.0)
            sim.advance(dt)
            sim.plasticUpdate(dt)
            sim.cleanUpV()
            sim.cleanUpAlpha()
            if sim.contains_nan():
                raise FloatingPointError("NaN in the state")
            dts.append(dt)
    else:
        sim.run(nsteps=case["steps"], t_end=1e300)
    for q in range(len(s.c.domains)):
        sim._check(sim.L.tj_download_domain(sim.h, q, _dp(s.out, s.out_at[q])))
    got = _fields(s, s.out)
    if case["do"] == "operators":
        got["dt"] = np.array(dts)
    return got


# ---------------------------------------------------------------------------
# What one pass cannot do without.
# ---------------------------------------------------------------------------
def work(case):
    kind = case["problem"]
    M, dim, solid = {"bubble": (2, 2, 0), "boxes": (2, 3, 0), "copper": (1, 3, 1), "solid_gas": (2, 2, 1),
                     "sod": (2, 1, 0)}[kind]
    if kind == "boxes":
        # edges log-uniform in [8, 64]: the mean edge cubed
        cells = case["n"] * (56.0 / math.log(8.0)) ** 3
    else:
        cells = float(case["n"]) ** dim
    w = 8 if case["precision"] == "fp64" else 4
    words = 3 * M + 2 * dim + 2 + (10 + 2 * M if solid else 0)  # carried state
    prim = 2 * M + 4 + (9 + M if solid else 0)
    ncomp = 3 * M + 18 + (28 + 2 * M if solid else 0)
    steps = case["steps"]
    # a stage reads its input and writes its output, the second also reads U^n
    per_step = 5 * words * w
    # reconstruction, closures, Riemann problem and update of one cell and direction, plus the closure of the stage
    per_stage = dim * (560 if solid else 210) + (420 if solid else 60)
    bytes_ = cells * (steps * per_step + 8 * (prim + ncomp))
    flops = cells * steps * 2.0 * per_stage
    if case["do"] == "exchange":
        bytes_ = cells * (per_step + 8.0 * (words + ncomp))
    elif case["do"] == "adjoint":  # forward, its recomputation, and a reverse sweep of at least twice the work
        bytes_, flops = bytes_ * 4.0, flops * 4.0
    elif case["do"] == "tangent":
        bytes_, flops = bytes_ * 2.0, flops * 3.0
    return {"bytes": bytes_, "flops": flops}


# ---------------------------------------------------------------------------
# The same update in 64 bits with plain torch: one face list per direction
# over all domains, gathers instead of ghost cells.
# ---------------------------------------------------------------------------
class _Plain:
    def __init__(self, c, device):
        self.c, self.M, self.dim = c, c.M, c.dim
        kw = dict(device=device)
        f64 = dict(dtype=torch.float64, device=device)
        N = self.N = sum(d.ncells for d in c.domains)
        shift = [-2, -1, 1, 2]
        near = {(d, o): [] for d in range(c.dim) for o in shift}
        flip = {(d, o): [] for d in range(c.dim) for o in shift}
        corner = {}
        dx = [[] for _ in range(3)]
        high, at = [[] for _ in range(3)], 0
        lo = [[] for _ in range(3)]
        hi = [[] for _ in range(3)]
        idx = [[] for _ in range(3)]

        def image(i, n, d):
            mirror_lo, mirror_hi = c.lo_bc[d] == 1, c.hi_bc[d] == 1
            m = np.where(i < 0, -1 - i if mirror_lo else 0, np.where(i > n - 1, 2 * n - 1 - i if mirror_hi else n - 1, i))
            return m, ((i < 0) & mirror_lo) | ((i > n - 1) & mirror_hi)

        for dom in c.domains:
            n = dom.n_cells
            k, j, i = np.meshgrid(*[np.arange(n[a]) for a in (2, 1, 0)], indexing="ij")
            ijk = [i.ravel(), j.ravel(), k.ravel()]

            def flat(p):
                return at + p[0] + n[0] * (p[1] + n[1] * p[2])

            for d in range(c.dim):
                for o in shift:
                    p = list(ijk)
                    p[d], f = image(ijk[d] + o, n[d], d)
                    near[d, o].append(flat(p))
                    flip[d, o].append(f)
                high[d].append(flat(ijk)[ijk[d] == n[d] - 1])
                dx[d].append(np.full(dom.ncells, dom.dim_l[d] / n[d]))
                idx[d].append(ijk[d])
            if c.thinc:
                for di in (-1, 0, 1):
                    for dj in (-1, 0, 1):
                        p = list(ijk)
                        p[0] = image(ijk[0] + di, n[0], 0)[0]
                        if c.dim > 1:
                            p[1] = image(ijk[1] + dj, n[1], 1)[0]
                        corner[di, dj] = torch.from_numpy(flat(p)).to(**kw)
                for d in range(3):
                    l, h = np.zeros(n[::-1], np.int64), np.zeros(n[::-1], np.int64)
                    for b in dom.boxes:
                        sl = (slice(b[2], b[5] + 1), slice(b[1], b[4] + 1), slice(b[0], b[3] + 1))
                        l[sl], h[sl] = b[d], b[3 + d]
                    lo[d].append(l.ravel())
                    hi[d].append(h.ravel())
            at += dom.ncells

        def put(v):
            return torch.from_numpy(np.concatenate(v)).to(**kw)

        self.near = {k: put(v) for k, v in near.items()}
        self.flip = {k: put(v) for k, v in flip.items()}
        self.corner = corner
        self.dx = [put(v) for v in dx[:c.dim]]
        own = torch.arange(N, **kw)
        self.left, self.right, self.lflip, self.rflip, self.upper = [], [], [], [], []
        for d in range(c.dim):
            hb = put(high[d])
            self.left.append(torch.cat([self.near[d, -1], hb]))
            self.right.append(torch.cat([own, hb]))
            self.lflip.append(torch.cat([self.flip[d, -1], torch.zeros_like(hb, dtype=torch.bool)]))
            self.rflip.append(torch.cat([torch.zeros(N, dtype=torch.bool, **kw), self.flip[d, 1][hb]]))
            u = self.near[d, 1].clone()
            u[hb] = N + torch.arange(len(hb), **kw)
            self.upper.append(u)
        q = [list(m.params) + [0.0] * 16 for m in c.materials]
        self.q = q
        self.G = [v[0] - 1.0 for v in q]
        self.is_solid = [m.phase == problems.PHASE_SOLID for m in c.materials]
        if c.thinc:
            self.ulstar = torch.zeros((self.M, N), **f64)
            self.urstar = torch.zeros((self.M, N), **f64)
            self.gstar = [torch.zeros((self.M, len(self.left[d])), **f64) for d in range(c.dim)]
            self.in_m = [put(idx[d]) - 1 >= put(lo[d]) for d in range(c.dim)]
            self.in_p = [put(idx[d]) + 1 <= put(hi[d]) for d in range(c.dim)]

    # -- closures ------------------------------------------------------------
    def cold(self, m, s, which):
        """Non-thermal energy ("e") or pressure ("p") of material m."""
        q, eos, G = self.q[m], self.c.materials[m].eos, self.G[m]
        if eos == problems.EOS_MIEGRUNEISEN:
            return q[2] * s["ar"][m] if which == "e" else q[1] * s["al"][m] / G
        x = s["rk"][m] / q[4]
        if eos == problems.EOS_WILKINS:
            shear = q[10]
            if which == "e":
                e = (q[5] + q[6] * x * x + q[7] * x + q[8] / x - q[9] * torch.log(x)) / q[4]
                return s["ar"][m] * e + s["al"][m] * shear * s["hj2"]
            pc = 2.0 * q[6] * x ** 3 + q[7] * x * x - q[8] - q[9] * x
            return s["al"][m] / G * (pc - shear * s["hj2"])
        et = 1.0 - 1.0 / x
        ph = q[4] * q[5] ** 2 * et / (1.0 - q[6] * et) ** 2
        if which == "e":
            return s["ar"][m] * ph * et / (2.0 * q[4]) + s["al"][m] * q[7] * s["hj2"]
        return s["al"][m] / G * (ph - q[7] * s["hj2"])

    def shear(self, m):
        return self.q[m][10 if self.c.materials[m].eos == problems.EOS_WILKINS else 7]

    def inv_gamma(self, s):
        return sum(s["al"][m] / self.G[m] for m in range(self.M))

    def strain(self, s):
        s["hj2"] = torch.zeros_like(s["rho"])
        if not self.c.solid:
            return
        V = s["V"].view(3, 3, -1)
        B = torch.einsum("ikn,jkn->ijn", V, V)
        s["devH"] = 0.25 * (B - _inv3(B))
        s["hj2"] = (s["devH"] ** 2).sum((0, 1))

    def stress(self, s):
        eye = torch.eye(3, dtype=torch.float64, device=s["p"].device)[:, :, None]
        s["sig"] = -s["p"] * eye
        if self.c.solid:
            g = sum(self.shear(m) * s["al"][m] / self.G[m] for m in range(self.M) if self.is_solid[m])
            s["sig"] = s["sig"] + 2.0 * (g / self.inv_gamma(s)) * s["devH"]

    def kinetic(self, s):
        return 0.5 * s["rho"] * (s["u"] ** 2).sum(0)

    def from_primitive(self, s):
        s["ar"] = s["al"] * s["rk"]
        s["rho"] = s["ar"].sum(0)
        if self.c.plastic:
            s["are"] = torch.stack([s["eps"][m] * s["ar"][m] if self.is_solid[m] else s["are"][m] for m in range(self.M)])
        self.strain(s)
        s["ru"] = s["u"] * s["rho"]
        nt = sum(self.cold(m, s, "e") - self.cold(m, s, "p") for m in range(self.M))
        s["E"] = s["p"] * self.inv_gamma(s) + nt + self.kinetic(s)
        self.stress(s)

    def from_conserved(self, s):
        s["rk"] = s["ar"] / s["al"]
        s["rho"] = s["ar"].sum(0)
        if self.c.plastic:
            s["eps"] = torch.stack([s["are"][m] / s["ar"][m] if self.is_solid[m] else s["eps"][m] for m in range(self.M)])
        self.strain(s)
        s["u"] = s["ru"] / s["rho"]
        s["p"] = torch.zeros_like(s["rho"])
        nt = sum(self.cold(m, s, "e") - self.cold(m, s, "p") for m in range(self.M))
        s["p"] = (s["E"] - self.kinetic(s) - nt) / self.inv_gamma(s)
        self.stress(s)

    def sound(self, s):
        tot, xit = 0.0, 0.0
        for m in range(self.M):
            q, G, r, p = self.q[m], self.G[m], s["rk"][m], s["p"]
            eos = self.c.materials[m].eos
            if eos == problems.EOS_MIEGRUNEISEN:
                c2 = (p * (G + 1.0) - q[1]) / r
            elif eos == problems.EOS_WILKINS:
                x = r / q[4]
                nt = self.cold(m, s, "p")
                c2 = (p - nt) * (G + 1.0) / r + (6.0 * q[6] * x * x + 2.0 * q[7] * x - q[9]) / q[4] + 4.0 / 3.0 * q[10] / r
            else:
                et = 1.0 - q[4] / r
                dd = 1.0 - q[6] * et
                k = q[4] * q[5] ** 2
                ph, dph, det = k * et / dd ** 2, k * (1.0 + q[6] * et) / dd ** 3, q[4] / r ** 2
                c2 = dph * det - G * r * (ph + et * dph) / (2.0 * q[4]) * det + (p * (G + 1.0) - ph) / r + 4.0 / 3.0 * q[7] / r
            tot = tot + torch.clamp(c2 * s["ar"][m] / s["rho"] / G, min=0.0)
            xit = xit + s["al"][m] / G
        tot = torch.where(tot <= 0.0, torch.full_like(tot, 1e-6), tot)
        return torch.sqrt(tot / xit)

    def clean_alpha(self, a):
        a = torch.where(a < 0.0, torch.full_like(a, 1e-6), torch.clamp(a, max=1.0))
        return a / a.sum(0)

    # -- reconstruction ------------------------------------------------------
    @staticmethod
    def limited(um, u0, up):
        r = (u0 - um) / (up - u0)
        r = torch.where(torch.isfinite(r), r, torch.zeros_like(r))
        lim = torch.where(r > 0.0, torch.minimum(2.0 * r, torch.full_like(r, 2.0)) / (1.0 + r), torch.zeros_like(r))
        half = 0.25 * lim * (up - um)
        return u0 - half, u0 + half

    def gather(self, w, d, o, row):
        v = w[:, self.near[d, o]]
        v[row] = torch.where(self.flip[d, o], -v[row], v[row])
        return v

    def thinc(self, al, d):
        aL, aR, eps = al[:, self.near[d, -1]], al[:, self.near[d, 1]], 1e-20
        mn, mx = torch.minimum(aL, aR), (aL - aR).abs()
        th = torch.sign(aR - aL)
        C = torch.where(mx < eps, torch.zeros_like(mx), (al - mn + eps) / (mx + eps))
        mixed = (C > 1e-4) & (C < 0.999999 - 1e-4) & ((aR - al) * (al - aL) >= 0.0)
        nv = torch.ones_like(al)
        if self.dim == 2:
            n = {k: al[:, i] for k, i in self.corner.items()}
            h = [dom / n_ for dom, n_ in zip(self.c.domains[0].dim_l, self.c.domains[0].n_cells)]
            gx = -(n[1, 1] + 2 * n[1, 0] + n[1, -1] - n[-1, 1] - 2 * n[-1, 0] - n[-1, -1]) / (8.0 * h[0])
            gy = -(n[1, 1] + 2 * n[0, 1] + n[-1, 1] - n[-1, -1] - 2 * n[0, -1] - n[1, -1]) / (8.0 * h[1])
            norm = torch.sqrt(gx * gx + gy * gy)
            nv = torch.where(norm < 1e-20, torch.zeros_like(norm), ((gx, gy)[d] / norm).abs())
        beta = nv * self.c.thinc_beta + 0.01
        tb = torch.tanh(beta)
        A = (torch.exp(th * beta * (2.0 * C - 1.0)) / torch.cosh(beta) - 1.0) / tb
        right = mn + 0.5 * mx * (1.0 + th * (tb + A) / (1.0 + A * tb))
        return mixed, mn + 0.5 * mx * (1.0 + th * A), right

    def reconstruct(self, s, d):
        M, c = self.M, self.c
        words = [s["al"], s["rk"], s["u"], s["p"][None]]
        if c.solid:
            words.append(s["V"])
        if c.plastic:
            words.append(s["eps"])
        w = torch.cat(words)
        lo, hi = self.limited(self.gather(w, d, -1, 2 * M + d), w, self.gather(w, d, 1, 2 * M + d))
        sides = [lo, hi]
        if c.thinc:
            al = s["al"]
            mixed, tl, tr = self.thinc(al, d)
            im, ip = self.near[d, -1], self.near[d, 1]
            in_m, in_p = self.in_m[d], self.in_p[d]
            tpl = torch.where(mixed, tl, self.ulstar)
            tpr = torch.where(mixed, tr, self.urstar)
            urm = torch.where(in_m, hi[:M][:, im], al[:, im])
            ulp = torch.where(in_p, lo[:M][:, ip], al[:, ip])
            trm = torch.where(in_m, tpr[:, im], torch.zeros_like(al))
            tlp = torch.where(in_p, tpl[:, ip], self.gstar[d][:, self.upper[d]])

            def tbv(a, b):
                pairs = [(urm, ulp), (trm, tlp), (urm, tlp), (trm, ulp)]
                return torch.stack([(x - a).abs() + (b - y).abs() for x, y in pairs]).amin(0)

            take = mixed[M - 1] & (tbv(tpl, tpr) < tbv(lo[:M], hi[:M]))
            lo[:M] = torch.where(take, tpl, lo[:M])
            hi[:M] = torch.where(take, tpr, hi[:M])
            self.ulstar = torch.where(mixed, tl, self.ulstar)
            self.urstar = torch.where(mixed, tr, self.urstar)
        out = []
        for v in sides:
            f = {"al": v[:M], "rk": v[M:2 * M], "u": v[2 * M:2 * M + 3], "p": v[2 * M + 3]}
            if c.solid:
                f["V"] = v[2 * M + 4:2 * M + 13]
            if c.plastic:
                f["eps"], f["are"] = v[-M:], s["are"]
            if c.thinc:
                f["al"] = self.clean_alpha(f["al"])
            self.from_primitive(f)
            f["a"] = self.sound(f)
            out.append(f)
        return out

    # -- Riemann problems ----------------------------------------------------
    def star(self, U, SK, S, d):
        ud = U["u"][d]
        mult = torch.where(((S - ud) / S).abs() < 1e-20, torch.ones_like(S), (SK - ud) / (SK - S))
        F = {"al": U["al"], "ar": mult * U["ar"], "ru": mult * U["ru"]}
        F["ru"][d] = mult * U["rho"] * S
        F["rho"] = F["ar"].sum(0)
        F["rk"] = F["ar"] / F["al"]
        F["u"] = F["ru"] / F["rho"]
        F["E"] = mult * U["rho"] * (U["E"] / U["rho"] + (S - ud) * (S - U["sig"][d, d] / (U["rho"] * (SK - ud))))
        if self.c.solid:
            F["V"] = mult * U["V"]
            F["V"][3 * d:3 * d + 3] = U["V"][3 * d:3 * d + 3]
        if self.c.plastic:
            F["are"] = torch.stack([mult * U["are"][m] * float(self.is_solid[m]) for m in range(self.M)])
        return F

    def vector(self, U):
        rows = [U["ar"], U["ru"], U["E"][None]]
        if self.c.solid:
            rows.append(U["V"])
        if self.c.plastic:
            rows.append(U["are"])
        return torch.cat(rows)

    def physical(self, U, d):
        ud = U["u"][d]
        rows = [U["ar"] * ud, U["ru"] * ud - U["sig"][:, d], (U["E"] * ud - (U["u"] * U["sig"][:, d]).sum(0))[None]]
        if self.c.solid:
            V = U["V"].view(3, 3, -1)
            rows.append((V * ud - V[d][None] * U["u"][:, None]).reshape(9, -1))
        if self.c.plastic:
            rows.append(U["are"] * ud)
        return torch.cat(rows)

    def transverse(self, F):
        inv = [F["al"][m] / self.G[m] for m in range(self.M)]
        b = sum(inv[m] * self.shear(m) / F["rk"][m] for m in range(self.M) if self.is_solid[m])
        b = torch.clamp(torch.nan_to_num(b, nan=0.0), min=0.0)
        return torch.nan_to_num(torch.sqrt(b / sum(inv)), nan=0.0)

    def fluxes(self, lo, hi, d):
        def take(f, at, fl):
            g = {k: v[..., at] for k, v in f.items()}
            for k in ("u", "ru"):
                g[k] = g[k].clone()
                g[k][d] = torch.where(fl, -g[k][d], g[k][d])
            return g

        L, R = take(hi, self.left[d], self.lflip[d]), take(lo, self.right[d], self.rflip[d])
        SR = torch.maximum(L["u"][d].abs() + L["a"], R["u"][d].abs() + R["a"])
        SL = -SR
        ml, mr = L["rho"] * (SL - L["u"][d]), R["rho"] * (SR - R["u"][d])
        S = (L["sig"][d, d] - R["sig"][d, d] + L["ru"][d] * (SL - L["u"][d]) - R["ru"][d] * (SR - R["u"][d])) / (ml - mr)
        Ls, Rs = self.star(L, SL, S, d), self.star(R, SR, S, d)
        left = (SL >= 0.0) | (S >= 0.0)
        fa = torch.where(left, Ls["al"] * Ls["u"][d], Rs["al"] * Rs["u"][d])
        qL, qR, qLs, qRs = self.vector(L), self.vector(R), self.vector(Ls), self.vector(Rs)
        pL, pR = self.physical(L, d), self.physical(R, d)
        fL, fR = pL + SL * (qLs - qL), pR + SR * (qRs - qR)
        vstar = None
        if self.c.solid:
            SLT, SRT = S - self.transverse(Ls), S + self.transverse(Rs)
            a, b = Ls["rho"] * (S - SLT), Rs["rho"] * (S - SRT)
            sg = (a * b * (L["u"] - R["u"]) + a * R["sig"][:, d] - b * L["sig"][:, d]) / (a - b)

            def inner(K, Ks, SKT):
                F = {k: v.clone() for k, v in Ks.items()}
                rows = [r for r in range(3) if r != d]
                for r in rows:
                    F["ru"][r] = F["ru"][r] + (sg[r] - K["sig"][r, d]) / (S - SKT)
                    F["u"][r] = F["ru"][r] / F["rho"]
                for r in rows:
                    F["E"] = F["E"] + (F["u"][r] * sg[r] - K["u"][r] * K["sig"][r, d]) / (S - SKT)
                    for q in range(3):
                        F["V"][3 * r + q] = F["V"][3 * r + q] + F["V"][3 * d + q] * (F["u"][r] - K["u"][r]) / (S - SKT)
                return F

            Lss, Rss = inner(L, Ls, SLT), inner(R, Rs, SRT)
            fL = torch.where(SLT >= 0.0, fL, fL + SLT * (self.vector(Lss) - qLs))
            fR = torch.where(SRT >= 0.0, fR + SRT * (self.vector(Rss) - qRs), fR)
            rows = slice(3 * d, 3 * d + 3)
            vL = torch.where(SL >= 0.0, L["V"][rows], torch.where(SLT >= 0.0, Ls["V"][rows], Lss["V"][rows]))
            vR = torch.where(SR < 0.0, R["V"][rows], torch.where(SRT >= 0.0, Rss["V"][rows], Rs["V"][rows]))
            vstar = torch.where(left, vL, vR)
        fL, fR = torch.where(SL >= 0.0, pL, fL), torch.where(SR >= 0.0, fR, pR)
        if self.c.thinc:
            src = torch.where(left, L["al"], R["al"])
            self.ulstar = src[:, :self.N].clone()
            edge = ~self.in_p[d]  # cells whose upper face leaves their box
            at = self.upper[d][edge]
            self.gstar[d][:, at] = src[:, at]
        return fa, torch.where(left, fL, fR), S, vstar

    # -- one step ------------------------------------------------------------
    def stage(self, s, dt):
        M, c = self.M, self.c
        q, al = self.vector(s).clone(), s["al"].clone()
        v0 = M + 4
        for d in range(self.dim):
            lo, hi = self.reconstruct(s, d)
            fa, f, S, vs = self.fluxes(lo, hi, d)
            up, k = self.upper[d], dt / self.dx[d]
            dS = S[:self.N] - S[up]
            al = al + k * (fa[:, :self.N] - fa[:, up] - s["al"] * dS)
            q = q + k * (f[:, :self.N] - f[:, up])
            if c.solid:
                dv = vs[:, :self.N] - vs[:, up]
                extra = s["u"][:, None] * dv[None] - (2.0 / 3.0) * s["V"].view(3, 3, -1) * dS
                q[v0:v0 + 9] += k * extra.reshape(9, -1)
        n = {"al": al, "ar": q[:M], "ru": q[M:M + 3], "E": q[M + 3]}
        if c.solid:
            n["V"] = q[v0:v0 + 9]
        if c.plastic:
            n["are"], n["eps"] = q[v0 + 9:], s["eps"]
        self.from_conserved(n)
        return n

    def dt(self, s):
        a = self.sound(s)
        return self.c.cfl * min(float((self.dx[d] / (a + s["u"][d].abs())).min()) for d in range(self.dim))

    def step(self, s, dt):
        two = self.stage(self.stage(s, dt), dt)
        keep = ["al", "ar", "rk", "rho", "ru", "u", "E", "p", "hj2"] + (["V"] if self.c.solid else []) + \
            (["eps", "are"] if self.c.plastic else [])
        n = {k: 0.5 * s[k] + 0.5 * two[k] for k in keep}
        if self.c.plastic:
            self.plastic(n)
            self.from_conserved(n)
        if self.c.solid:
            V = n["V"].view(3, 3, -1)
            root = _sqrt3(torch.einsum("ikn,jkn->ijn", V, V))
            ts = sum(n["al"][m] for m in range(self.M) if self.is_solid[m])
            ta = n["al"].sum(0)
            eye = torch.eye(3, dtype=torch.float64, device=V.device)[:, :, None]
            n["V"] = ((root * _det3(root) ** (-1.0 / 3.0) * ts + eye * (ta - ts)) / ta).reshape(9, -1)
        n["al"] = self.clean_alpha(n["al"])
        return n

    def plastic(self, n):
        ts = sum(n["al"][m] for m in range(self.M) if self.is_solid[m])
        fluid = ts <= 0.5
        self.strain(n)
        J = torch.sqrt(n["hj2"])
        JB, JT = torch.zeros_like(J), torch.zeros_like(J)
        eps, are = torch.zeros_like(n["eps"]), torch.zeros_like(n["are"])
        for m in range(self.M):
            if not self.is_solid[m]:
                continue
            cap = self.c.materials[m].yield_stress / (math.sqrt(3.0) * self.shear(m))
            Jn = torch.clamp(J, max=cap)
            eps[m] = torch.where(fluid, torch.zeros_like(J), n["eps"][m] + math.sqrt(2.0 / 3.0) * (J - Jn))
            are[m] = eps[m] * n["ar"][m]
            JB, JT = JB + n["al"][m] / self.G[m] * J, JT + n["al"][m] / self.G[m] * Jn
        none = JB == 0.0
        k = torch.where(none, torch.ones_like(JB), JT / torch.where(none, torch.ones_like(JB), JB))
        eye = torch.eye(3, dtype=torch.float64, device=J.device)[:, :, None]
        dev = n["devH"] * k
        V = torch.einsum("ikn,kjn->ijn", _inv3(eye - 0.5 * dev), eye + 0.5 * dev).reshape(9, -1)
        n["eps"], n["are"], n["V"] = eps, are, torch.where(fluid, n["V"], V)

    def initial(self):
        """The initial state of the primitive fields (primitiveToConservative)."""
        c, M = self.c, self.M
        prim = torch.from_numpy(np.concatenate([d.prim.reshape(c.nprim, -1) for d in c.domains], axis=1))
        prim = prim.to(self.dx[0].device)
        s = {"al": prim[:M], "rk": prim[M:2 * M], "u": prim[2 * M:2 * M + 3], "p": prim[2 * M + 3]}
        if c.solid:
            s["V"] = prim[2 * M + 4:2 * M + 13]
        if c.plastic:
            s["eps"], s["are"] = prim[2 * M + 13:2 * M + 13 + M], torch.zeros_like(prim[:M])
        self.from_primitive(s)
        return s

    def fields(self, s, precision):
        """The state, laid out as run() returns it."""
        c, M = self.c, self.M
        parts = {"alpha": s["al"], "alpha_rho": s["ar"], "momentum": s["ru"], "velocity": s["u"],
                 "energy": s["E"][None], "pressure": s["p"][None]}
        if precision == "fp64":
            parts["rho_k"] = s["rk"]
        if c.solid:
            parts["strain"] = torch.cat([s["V"], s["hj2"][None]] + ([s["eps"]] if c.plastic else []))
        if c.plastic:
            parts["alpha_rho_strain"] = torch.cat([parts.pop("alpha_rho"), s["are"]])
        cells = [d.ncells for d in c.domains]
        if len(cells) == 1:
            return {k: v.reshape((-1,) + tuple(c.domains[0].n_cells[::-1])) for k, v in parts.items()}
        return {k: torch.cat([p.reshape(-1) for p in v.split(cells, dim=1)]) for k, v in parts.items()}


def _det3(A):
    return (A[0, 0] * (A[1, 1] * A[2, 2] - A[1, 2] * A[2, 1]) - A[0, 1] * (A[1, 0] * A[2, 2] - A[1, 2] * A[2, 0]) +
            A[0, 2] * (A[1, 0] * A[2, 1] - A[1, 1] * A[2, 0]))


def _inv3(A):
    a = torch.roll(A, (-1, -1), (0, 1)) * torch.roll(A, (-2, -2), (0, 1))
    b = torch.roll(A, (-1, -2), (0, 1)) * torch.roll(A, (-2, -1), (0, 1))
    return (a - b).transpose(0, 1) / _det3(A)


def _sqrt3(A):
    """Square root of symmetric positive definite 3x3 matrices (Denman and Beavers' iteration)."""
    Y, Z = A, torch.eye(3, dtype=torch.float64, device=A.device)[:, :, None].expand_as(A)
    for _ in range(8):
        Y, Z = 0.5 * (Y + _inv3(Z)), 0.5 * (Z + _inv3(Y))
    return Y


def exact(case, seed):
    c = _problem(case, seed)
    plain = _Plain(c, "cuda" if torch.cuda.is_available() else "cpu")
    s = plain.initial()
    dts = []
    for n in range(case["steps"]):
        dt = plain.dt(s)
        dts.append(dt * 0.2 if n < 5 else dt)
        s = plain.step(s, dts[-1])
    got = plain.fields(s, case["precision"])
    if case["do"] == "operators":
        got["dt"] = np.array(dts)
    if case["do"] == "adjoint":  # the derivatives follow the update's own branches at its kinks
        return {"state": got, "grad_prim": None, "grad_eos": None}
    if case["do"] == "tangent":
        return {"state": got, "tangent": None}
    return got
