"""The solver calls whose speed this framework is measured by.

Each case is one call pattern of a user's program: the right-hand side alone
(a program with its own time integrator), a run of SSPRK3 steps from a given
state, the gradient of an objective through a run, and a batch of meshes
advanced by a captured graph.  Together they cover both dimensions, every
two-point and surface flux, shock capturing, the viscous terms, powers of two
and odd degrees and element counts, meshes from a few hundred nodes (a launch
is most of the time) to 16 million (states stream from memory), and solvers
used as constructed as well as solvers that tune their launch shape first,
which programs with long runs do.

`exact` is the method written out in plain torch on uniform Cartesian
elements, in 64 bits and without this package's code: per direction d
    du -= 2/h_d [ sum_k 2 D_mk f#(u_m, u_k) + (delta_mN f*_hi - delta_m0 f*_lo) / w_m ]
with the subcell blend, the viscous terms and the boundary states around it.
"""
import math
import random

import numpy as np
import torch

import dgsem_b200 as D

GAMMA = 1.4
MU, PRANDTL = 1.0e-3, 0.72

DOMAIN = {"kh": (-1.0, 1.0), "vortex": (-5.0, 5.0), "tgv": (0.0, 2.0 * math.pi),
          "tgv2d": (0.0, 2.0 * math.pi)}
# largest |v| + c of each flow, for the time step
SPEED = {"kh": 1.9, "vortex": 4.0, "tgv": 11.5, "tgv2d": 11.5, "dmr": 12.0}


def _case(name, op, flow, polydeg, nx, ny, nz, vf, sf="llf", hg=False, viscous=False, steps=1,
          tuned=False, meshes=1):
    c = dict(op=op, flow=flow, polydeg=polydeg, nx=nx, ny=ny, nz=nz, vf=vf, sf=sf, hg=hg,
             viscous=viscous, steps=steps, tuned=tuned, meshes=meshes)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # one right-hand side on a mesh of a test or a tutorial: launch and
        # latency only; the shear layer with shock capturing
        _case("rhs_kh_16x16_hg", "rhs", "kh", 3, 16, 16, 0, "chandrashekar", hg=True),
        # the 2D benchmark configuration, stepped call by call
        _case("kh_64x64", "steps", "kh", 3, 64, 64, 0, "ranocha", steps=10, tuned=True),
        # a production 2D mesh whose states do not fit in L2
        _case("kh_1024x1024", "steps", "kh", 3, 1024, 1024, 0, "ranocha", steps=4, tuned=True),
        # the 3D benchmark configuration
        _case("tgv_16", "steps", "tgv", 3, 16, 16, 16, "kennedy_gruber", steps=10, tuned=True),
        # a larger 3D box with the entropy-conservative flux, solver as constructed
        _case("tgv_32_ec", "steps", "tgv", 3, 32, 32, 32, "chandrashekar", steps=4),
        # double Mach reflection: shock capturing, HLLC, time-dependent boundaries
        _case("dmr_240x60", "steps", "dmr", 3, 240, 60, 0, "chandrashekar", sf="hllc", hg=True,
              steps=10, tuned=True),
        # ragged element counts and an odd degree, solver as constructed
        _case("vortex_97x61_n6", "steps", "vortex", 5, 97, 61, 0, "chandrashekar", steps=6),
        # 3D shock capturing at five nodes per direction, ragged counts
        _case("tgv_hg_11x9x13_n5", "steps", "tgv", 4, 11, 9, 13, "chandrashekar", hg=True,
              steps=6),
        # viscous shear layer with shock capturing (2D Navier-Stokes)
        _case("khv_80x72_n5", "steps", "kh", 4, 80, 72, 0, "chandrashekar", hg=True,
              viscous=True, steps=6),
        # viscous Taylor-Green vortex (3D Navier-Stokes)
        _case("tgv_ns_16", "steps", "tgv", 3, 16, 16, 16, "chandrashekar", viscous=True, steps=6),
        # gradient of the kinetic energy through 40 Navier-Stokes steps
        _case("adjoint_32x32_n5", "gradient", "tgv2d", 4, 32, 32, 0, "chandrashekar",
              viscous=True, steps=40, tuned=True),
        # an ensemble of vortices on uneven meshes and degrees, one captured step
        _case("batch_64", "batch", "vortex", 0, 0, 0, 0, "chandrashekar", steps=2, tuned=True,
              meshes=64),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choice(["euler2d"] * 4 + ["euler3d"] * 3 + ["dmr", "ns2d", "ns3d", "adjoint",
                                                             "batch"])
    tuned = rng.random() < 0.5
    steps = rng.randint(2, 10)
    op = "rhs" if rng.random() < 0.25 else "steps"
    fluxes = ["chandrashekar", "ranocha", "kennedy_gruber"]
    if family == "euler2d":
        deg = rng.choice([1, 2, 3, 3, 3, 4, 5, 6, 7])
        top = int(1000 / (deg + 1))
        nx, ny = _log_int(rng, 6, top), _log_int(rng, 6, top)
        vf, sf, hg = rng.choice(fluxes), "llf", rng.random() < 0.3
        if deg == 3:
            sf = rng.choice(["llf", "llf", "hllc"])
        elif hg:
            vf = "chandrashekar"
        return _case(None, op, rng.choice(["kh", "vortex"]), deg, nx, ny, 0, vf, sf, hg,
                     steps=steps, tuned=tuned)
    if family == "euler3d":
        deg = rng.choice([1, 2, 3, 3, 4])
        top = int(120 / (deg + 1))
        n3 = [_log_int(rng, 4, top) for _ in range(3)]
        vf, hg = rng.choice(fluxes), rng.random() < 0.25
        if hg and deg != 3:
            vf = "chandrashekar"
        return _case(None, op, "tgv", deg, *n3, vf, "llf", hg, steps=steps, tuned=tuned)
    if family == "dmr":
        ny = _log_int(rng, 12, 120)
        return _case(None, op, "dmr", 3, 4 * ny + rng.randint(-3, 3), ny, 0,
                     rng.choice(fluxes), rng.choice(["llf", "hllc"]), True, steps=steps,
                     tuned=tuned)
    if family == "ns2d":
        deg = rng.randint(1, 7)
        top = int(500 / (deg + 1))
        nx, ny = _log_int(rng, 6, top), _log_int(rng, 6, top)
        return _case(None, op, "kh", deg, nx, ny, 0, "chandrashekar", hg=rng.random() < 0.5,
                     viscous=True, steps=steps, tuned=tuned)
    if family == "ns3d":
        deg = rng.randint(1, 4)
        top = int(80 / (deg + 1))
        n3 = [_log_int(rng, 4, top) for _ in range(3)]
        return _case(None, op, "tgv", deg, *n3, rng.choice(fluxes), viscous=True, steps=steps,
                     tuned=tuned)
    if family == "adjoint":
        deg = rng.randint(1, 5)
        nx, ny = _log_int(rng, 6, 48), _log_int(rng, 6, 48)
        return _case(None, "gradient", "tgv2d", deg, nx, ny, 0, "chandrashekar",
                     viscous=rng.random() < 0.7, steps=rng.randint(10, 40), tuned=tuned)
    return _case(None, "batch", "vortex", 0, 0, 0, 0, "chandrashekar", steps=rng.randint(1, 2),
                 tuned=tuned, meshes=_log_int(rng, 4, 60))


# ---------------------------------------------------------------- sizes
def _cells(case):
    return (case["nx"], case["ny"]) + ((case["nz"],) if case["nz"] else ())


def _box(case):
    """(left, right) per axis."""
    dim = len(_cells(case))
    if case["flow"] == "dmr":
        return (0.0, 0.0), (4.0, 1.0)
    lo, hi = DOMAIN[case["flow"]]
    return (lo,) * dim, (hi,) * dim


def _dt(case):
    cells, (lo, hi) = _cells(case), _box(case)
    h = min((hi[a] - lo[a]) / cells[a] for a in range(len(cells)))
    cfl = 0.3 if len(cells) == 3 else 0.4
    dt = cfl * h / ((2.0 * case["polydeg"] + 1.0) * SPEED[case["flow"]])
    if case["viscous"]:
        dt = min(dt, 0.05 * h * h / ((case["polydeg"] + 1.0) ** 4 * MU))
    return dt


def _batch_members(case):
    """The meshes of a batch: 16..128 squared elements, degrees 2..7."""
    rng = random.Random(1000 + case["meshes"])
    out = []
    for _ in range(case["meshes"]):
        k = rng.randint(16, 128)
        out.append(_case(None, "steps", "vortex", rng.randint(2, 7), k, k, 0, case["vf"],
                         steps=case["steps"]))
    return out


# ---------------------------------------------------------------- inputs
def _nodes(deg):
    """Legendre-Gauss-Lobatto nodes and weights."""
    c = np.zeros(deg + 1)
    c[deg] = 1.0
    leg = np.polynomial.legendre.Legendre(c)
    d1, d2 = leg.deriv(1), leg.deriv(2)
    x = np.sort(np.real(d1.roots())) if deg > 1 else np.zeros(0)
    for _ in range(4):
        x = x - d1(x) / d2(x)
    x = 0.5 * (x - x[::-1])
    x = np.concatenate([[-1.0], x, [1.0]])
    return x, 2.0 / (deg * (deg + 1.0) * leg(x) ** 2)


def _axes(case, dev):
    """Node coordinates per axis, shaped to broadcast over (elements..., nodes...)."""
    cells, (lo, hi) = _cells(case), _box(case)
    dim, x = len(cells), _nodes(case["polydeg"])[0]
    out = []
    for a in range(dim):
        dx = 2.0 / cells[a]
        c = (-1.0 + np.arange(cells[a]) * dx + 0.5 * dx)[:, None] + 0.5 * dx * x[None, :]
        pos = torch.from_numpy(0.5 * ((1.0 - c) * lo[a] + (1.0 + c) * hi[a])).to(dev)
        shape = [1] * (2 * dim)
        shape[dim - 1 - a], shape[2 * dim - 1 - a] = pos.shape
        out.append(pos.view(shape))
    return out


def _waves(xs, lo, hi, g):
    """A smooth periodic field of size 1 with random phases."""
    total = 0.0
    for _ in range(3):
        arg = 2.0 * math.pi * float(torch.rand((), generator=g, dtype=torch.float64))
        for a, x in enumerate(xs):
            arg = arg + int(torch.randint(0, 3, (), generator=g)) * 2.0 * math.pi * (
                x - lo[a]) / (hi[a] - lo[a])
        total = total + (torch.sin(arg) if torch.is_tensor(arg) else math.sin(arg))
    return total / 3.0


def _primitive(case, xs, g):
    """rho, velocities and p of the flow with a seeded perturbation."""
    lo, hi = _box(case)
    flow = case["flow"]
    rnd = lambda: float(torch.rand((), generator=g, dtype=torch.float64))
    w = [_waves(xs, lo, hi, g) for _ in range(3)]
    x, y = xs[0], xs[1]
    if flow == "kh":
        b = torch.tanh(15.0 * y + 7.5) - torch.tanh(15.0 * y - 7.5)
        rho = 0.5 + 0.75 * b
        v = [0.5 * (b - 1.0) + 0.01 * w[0],
             0.1 * torch.sin(2.0 * math.pi * (x + rnd())) + 0.01 * w[1]]
        p = 1.0 + 0.02 * w[2]
    elif flow == "vortex":
        beta, dx, dy = 2.0 + 4.0 * rnd(), x - (4.0 * rnd() - 2.0), y - (4.0 * rnd() - 2.0)
        r2 = dx * dx + dy * dy
        e = beta / (2.0 * math.pi) * torch.exp(0.5 * (1.0 - r2))
        temp = 1.0 - (GAMMA - 1.0) / (2.0 * GAMMA) * e * e
        rho = temp ** (1.0 / (GAMMA - 1.0))
        v = [1.0 - e * dy, e * dx]
        p = rho * temp
    elif flow == "dmr":
        post = x < 1.0 / 6.0 + y / math.sqrt(3.0)
        one = torch.ones_like(x + y)
        pick = lambda a, b: torch.where(post, a * one, b * one)
        rho = pick(8.0, 1.4) * (1.0 + 0.01 * w[0])
        v = [pick(8.25 * math.cos(math.pi / 6.0), 0.0), pick(-8.25 * math.sin(math.pi / 6.0), 0.0)]
        p = pick(116.5, 1.0) * (1.0 + 0.01 * w[1])
    elif flow == "tgv":
        z = xs[2]
        rho = 1.0 + 0.01 * w[0]
        v = [torch.sin(x) * torch.cos(y) * torch.cos(z) + 0.01 * w[1],
             -torch.cos(x) * torch.sin(y) * torch.cos(z) + 0.01 * w[2], 0.05 * w[1]]
        p = 100.0 / 1.4 + (torch.cos(2 * x) + torch.cos(2 * y)) * (torch.cos(2 * z) + 2.0) / 16.0
    else:
        rho = 1.0 + 0.01 * w[0]
        v = [torch.sin(x) * torch.cos(y), -torch.cos(x) * torch.sin(y)]
        p = 100.0 / 1.4 + (torch.cos(2 * x) + torch.cos(2 * y)) / 4.0 + 0.1 * w[1]
    return rho, v, p


def _state(case, seed, dev):
    """Conserved state in the solver's layout u[element][variable][node]."""
    g = torch.Generator().manual_seed(seed)
    cells, n = _cells(case), case["polydeg"] + 1
    dim = len(cells)
    xs = _axes(case, dev)
    rho, v, p = _primitive(case, xs, g)
    shape = tuple(reversed(cells)) + (n,) * dim
    energy = p / (GAMMA - 1.0) + 0.5 * rho * sum(c * c for c in v)
    u = torch.stack([f.expand(shape) for f in [rho] + [rho * c for c in v] + [energy]])
    if case["flow"] == "tgv2d":  # nodal noise on the momentum
        noise = torch.randn((2,) + shape, generator=g, dtype=torch.float64)
        u[1:3] += 1.0e-3 * noise.to(dev)
    return u.movedim(0, dim).reshape(math.prod(cells), dim + 2, n ** dim).contiguous()


# ---------------------------------------------------------------- the framework's calls
def _solver(case):
    cells, (lo, hi) = _cells(case), _box(case)
    dim = len(cells)
    if case["viscous"]:
        cls = D.CompressibleNavierStokes2D if dim == 2 else D.CompressibleNavierStokes3D
        eq = cls(GAMMA, MU, PRANDTL)
    else:
        eq = D.CompressibleEuler2D(GAMMA) if dim == 2 else D.CompressibleEuler3D(GAMMA)
    vf = {"chandrashekar": D.ChandrashekarFlux, "ranocha": D.RanochaFlux,
          "kennedy_gruber": D.KennedyGruberFlux}[case["vf"]]
    sf = {"llf": D.LaxFriedrichsFlux, "hllc": D.HLLCFlux}[case["sf"]]
    vi = (D.VolumeIntegralShockCapturingHG if case["hg"] else D.VolumeIntegralSplitForm)(vf)
    if case["flow"] == "dmr":
        bcs = D.BoundarySet(D.DirichletBC("double_mach"), D.OutflowBC(),
                            D.MixedDirichletSlipWallBC("double_mach"),
                            D.DirichletBC("double_mach"))
    else:
        bcs = D.BoundarySet(*[D.PeriodicBC() for _ in range(2 * dim)])
    mesh = D.StructuredMesh(lo, hi, cells)
    basis = D.LobattoLegendreBasis(case["polydeg"])
    return eq, basis, mesh, D.StructuredSolver(eq, basis, vi, sf(), mesh, bcs)


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    if case["op"] == "batch":
        members = _batch_members(case)
        batch = D.BatchSolver(D.CompressibleEuler2D(GAMMA),
                              [(D.StructuredMesh(*_box(m), _cells(m)), m["polydeg"])
                               for m in members])
        u0 = torch.cat([_state(m, 1000 * seed + k, dev).reshape(-1)
                        for k, m in enumerate(members)])
        dts = [_dt(m) for m in members]
        batch.u.copy_(u0)
        if case["tuned"]:
            batch.autotune(dts)
        return dict(case=case, u0=u0, batch=batch, graph=batch.graph(dts, case["steps"]))
    eq, basis, mesh, solver = _solver(case)
    sol = D.Solution(mesh, basis, eq)
    u0 = _state(case, seed, dev)
    sol.u.copy_(u0)
    if case["tuned"]:
        solver.autotune(u0)
    state = dict(case=case, u0=u0, solver=solver, sol=sol, mesh=mesh, dt=_dt(case))
    if case["op"] == "steps":
        state["integrator"] = D.SSPRK3(sol, mesh)
    elif case["op"] == "gradient":
        state["adjoint"] = D.Adjoint(solver, case["steps"], checkpoint_every=20)
    return state


def run(state):
    op = state["case"]["op"]
    if op == "rhs":
        state["solver"].calc_rhs(state["sol"], 0.0)
        return state["sol"].rhs()
    if op == "gradient":
        return state["adjoint"].gradient(state["u0"], 0.0, state["dt"])
    if op == "batch":
        state["batch"].u.copy_(state["u0"])
        state["graph"].launch()
        return state["batch"].u
    sol, integ = state["sol"], state["integrator"]
    sol.u.copy_(state["u0"])
    integ.time = 0.0
    integ.solve_steps(state["solver"], sol, state["dt"], state["case"]["steps"])
    return sol.state()


# ---------------------------------------------------------------- work and tolerance
def work(case):
    """State in and state (or right-hand side) out; arithmetic per node and
    right-hand side: n - 1 two-point fluxes per direction shared by two nodes
    with their accumulation, 2 dim / n face fluxes shared by two elements, the
    node's primitive variables, and the stage combination.  A quotient, root
    or logarithm counts as one operation."""
    if case["op"] == "batch":
        parts = [work(m) for m in _batch_members(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    cells, n = _cells(case), case["polydeg"] + 1
    dim, nv = len(cells), len(cells) + 2
    nodes = math.prod(cells) * n ** dim
    pair = {"kennedy_gruber": 9 * dim + 9, "chandrashekar": 11 * dim + 34,
            "ranocha": 10 * dim + 36}[case["vf"]] + 4 * nv
    face = {"llf": 20 * dim + 24, "hllc": 110}[case["sf"]]
    per_node = dim * (n - 1) / 2 * pair + dim / n * face + 4 * dim + 8 + 6 * nv
    if case["hg"]:
        per_node += 2 * dim * n + 8
    if case["viscous"]:
        per_node += dim * (4 * n * (nv - 1) + 4 * nv) + 12 * dim * dim
    evals = 3 * case["steps"] if case["op"] != "rhs" else 1
    if case["op"] == "gradient":
        evals *= 3  # forward, and the reverse sweep at twice its operations
    return {"bytes": 2.0 * 8.0 * nv * nodes, "flops": float(evals * nodes * per_node)}


def tolerance(case):
    """About four times the distance to `exact` over the ranges.  A right-hand
    side is a small difference of large fluxes divided by the element size
    (seen: up to 2.8e-11); a few steps add it with the time step (4e-14); the
    gradient passes through every step twice (3e-13 at 40 steps)."""
    if case["op"] == "rhs":
        return {"rel": 1.2e-10}
    if case["op"] == "gradient":
        return {"rel": 2.0e-12}
    return {"rel": 2.0e-13}


# ---------------------------------------------------------------- the method in plain torch
class _Method:
    def __init__(self, case, dev):
        self.case, self.dev = case, dev
        self.cells, self.n = _cells(case), case["polydeg"] + 1
        self.dim = len(self.cells)
        lo, hi = _box(case)
        self.h = [(hi[a] - lo[a]) / self.cells[a] for a in range(self.dim)]
        x, w = _nodes(case["polydeg"])
        n = self.n
        bary = [1.0 / np.prod([x[j] - x[k] for k in range(n) if k != j]) for j in range(n)]
        d = np.array([[bary[j] / bary[i] / (x[i] - x[j]) if i != j else 0.0 for j in range(n)]
                      for i in range(n)])
        d -= np.diag(d.sum(1))
        self.w, self.d = w, d
        self.dhat = -(d.T * w[None, :]) / w[:, None]
        vand = np.stack([np.polynomial.legendre.Legendre.basis(k)(x) * math.sqrt(k + 0.5)
                         for k in range(n)], 1)
        self.vinv = torch.from_numpy(np.linalg.inv(vand)).to(dev)

    def node_axis(self, d):
        return -1 - d

    def elem_axis(self, d):
        return -1 - self.dim - d

    def split(self, u):
        """[E][var][node] -> one tensor per variable, (elements..., nodes...)."""
        shape = tuple(reversed(self.cells)) + (self.dim + 2,) + (self.n,) * self.dim
        return list(u.reshape(shape).unbind(self.dim))

    def join(self, parts):
        return torch.stack(parts, self.dim).reshape(
            math.prod(self.cells), self.dim + 2, self.n ** self.dim)

    def prim(self, u):
        """(conserved list, velocities, pressure)."""
        v = [m / u[0] for m in u[1:-1]]
        p = (GAMMA - 1.0) * (u[-1] - 0.5 * u[0] * sum(c * c for c in v))
        return u, v, p

    @staticmethod
    def log_mean(a, b):
        f2 = ((a - b) / (a + b)) ** 2
        small = f2 < 1.0e-4
        series = (a + b) / (2.0 + f2 * (2.0 / 3.0 + f2 * (2.0 / 5.0 + f2 * (2.0 / 7.0))))
        b2 = torch.where(small, 2.0 * a, b)  # keeps the unused branch finite
        return torch.where(small, series, (b2 - a) / torch.log(b2 / a))

    def volume_flux(self, left, right, d):
        (uL, vL, pL), (uR, vR, pR) = left, right
        dim, kind = self.dim, self.case["vf"]
        va = [0.5 * (a + b) for a, b in zip(vL, vR)]
        if kind == "kennedy_gruber":
            rho, p = 0.5 * (uL[0] + uR[0]), 0.5 * (pL + pR)
            e = 0.5 * (uL[-1] / uL[0] + uR[-1] / uR[0])
            f1 = rho * va[d]
            energy = (rho * e + p) * va[d]
        elif kind == "chandrashekar":
            bL, bR = 0.5 * uL[0] / pL, 0.5 * uR[0] / pR
            f1 = self.log_mean(uL[0], uR[0]) * va[d]
            p = 0.5 * (uL[0] + uR[0]) / (bL + bR)
            kin = 0.5 * (sum(c * c for c in vL) + sum(c * c for c in vR))
            energy = f1 * 0.5 * (1.0 / ((GAMMA - 1.0) * self.log_mean(bL, bR)) - kin)
            energy = energy + sum((f1 * va[c] + (p if c == d else 0.0)) * va[c]
                                  for c in range(dim))
        else:
            f1 = self.log_mean(uL[0], uR[0]) * va[d]
            p = 0.5 * (pL + pR)
            ratio = pL * pR / self.log_mean(uL[0] * pR, uR[0] * pL)
            dot = sum(a * b for a, b in zip(vL, vR))
            energy = f1 * (0.5 * dot + ratio / (GAMMA - 1.0)) + 0.5 * (pL * vR[d] + pR * vL[d])
        return [f1] + [f1 * va[c] + (p if c == d else 0.0) for c in range(dim)] + [energy]

    def physical_flux(self, s, d):
        u, v, p = s
        f = [c * v[d] for c in u]
        f[1 + d] = f[1 + d] + p
        f[-1] = f[-1] + p * v[d]
        return f

    def llf(self, left, right, d):
        (uL, vL, pL), (uR, vR, pR) = left, right
        aL, aR = torch.sqrt(GAMMA * pL / uL[0]), torch.sqrt(GAMMA * pR / uR[0])
        lam = torch.maximum(vL[d].abs(), vR[d].abs()) + torch.maximum(aL, aR)
        return [0.5 * (a + b) - 0.5 * lam * (y - x) for a, b, x, y in
                zip(self.physical_flux(left, d), self.physical_flux(right, d), uL, uR)]

    def hllc(self, left, right, d):
        (uL, vL, pL), (uR, vR, pR) = left, right
        e = 1 - d
        n1, n2, w1, w2 = vL[d], vR[d], vL[e], vR[e]
        cL, cR = torch.sqrt(GAMMA * pL / uL[0]), torch.sqrt(GAMMA * pR / uR[0])
        sL, sR = torch.sqrt(uL[0]), torch.sqrt(uR[0])
        roe = lambda a, b: (sL * a + sR * b) / (sL + sR)
        v, w = roe(n1, n2), roe(w1, w2)
        H = roe((uL[-1] + pL) / uL[0], (uR[-1] + pR) / uR[0])
        c = torch.sqrt((GAMMA - 1.0) * (H - 0.5 * (v * v + w * w)))
        SL, SR = torch.minimum(n1 - cL, v - c), torch.maximum(n2 + cR, v + c)
        qL, qR = uL[0] * (SL - n1), uR[0] * (SR - n2)
        SM = (pR - pL + qL * n1 - qR * n2) / (qL - qR)
        fL, fR = self.physical_flux(left, d), self.physical_flux(right, d)

        def star(u, f, S, q, vn, wt, p):
            rho = q / (S - SM)
            en = u[-1] / u[0] + (SM - vn) * (SM + p / q)
            us = [rho, None, None, rho * en]
            us[1 + d], us[1 + e] = rho * SM, rho * wt
            return [a + S * (b - x) for a, b, x in zip(f, us, u)]

        gL, gR = star(uL, fL, SL, qL, n1, w1, pL), star(uR, fR, SR, qR, n2, w2, pR)
        return [torch.where(SL >= 0.0, a, torch.where(SR <= 0.0, b, torch.where(SM >= 0.0, x, y)))
                for a, b, x, y in zip(fL, fR, gL, gR)]

    def surface_flux(self, left, right, d):
        return (self.hllc if self.case["sf"] == "hllc" else self.llf)(left, right, d)

    def at(self, s, d, m):
        """The state s at node m of every line along d."""
        ax = self.node_axis(d)
        pick = lambda f: f.select(ax, m)
        return [pick(f) for f in s[0]], [pick(f) for f in s[1]], pick(s[2])

    def alpha(self, u):
        """Hennemann-Gassner blending factor per element."""
        n, dim = self.n, self.dim
        v = [m / u[0] for m in u[1:-1]]
        ind = (1.4 - 1.0) * (u[-1] - 0.5 * u[0] * sum(c * c for c in v)) * u[0]
        for d in range(dim):
            ind = torch.movedim(torch.tensordot(ind, self.vinv, ([ind.dim() - 1 - d], [1])),
                                -1, ind.dim() - 1 - d)
        e = ind * ind
        sub = lambda k: e[(Ellipsis,) + (slice(0, max(k, 0)),) * dim].flatten(-dim).sum(-1)
        c1, c2 = sub(n - 1), sub(n - 2)
        if dim == 2:
            total = sub(n)
        else:  # the indicator's 3D total covers the layer k = N and the rows j = N
            total = c1 + e[..., n - 1, :, :].sum((-1, -2)) + e[..., : n - 1, n - 1, :].sum((-1, -2))
        zero = torch.zeros_like(total)
        e1 = torch.where(total != 0.0, (total - c1) / total, zero)
        e2 = torch.where(c1 != 0.0, (c1 - c2) / c1, zero)
        thr = 0.5 * 10.0 ** (-1.8 * n ** 0.25)
        s = math.log((1.0 - 1.0e-4) / 1.0e-4)
        a = 1.0 / (1.0 + torch.exp(-s / thr * (torch.maximum(e1, e2) - thr)))
        a = torch.where(a < 1.0e-3, zero, a).clamp(max=0.5)
        return a[(Ellipsis,) + (None,) * (dim - 1)]

    def gradient(self, q, d, lift):
        """Lifted derivative of q along d (2/h)(sum_k Dhat q_k + faces)."""
        ax, n = self.node_axis(d), self.n
        lines = q.unbind(ax)
        out = [sum(float(self.dhat[m, k]) * lines[k] for k in range(n)) for m in range(n)]
        hi, lo = lift
        out[n - 1] = out[n - 1] + hi / float(self.w[n - 1])
        out[0] = out[0] - lo / float(self.w[0])
        return torch.stack(out, ax) * (2.0 / self.h[d])

    def viscous(self, u, v, p):
        """-F_v per direction (lists of variables) from the BR1 gradient."""
        dim, q = self.dim, list(v) + [p / u[0]]
        grad = []
        for d in range(dim):
            # face traces: one position per line, so the element axis sits one
            # place further right for each node axis that is gone
            ea = self.elem_axis(d) + 1
            g = []
            for f in q:
                hi = f.select(self.node_axis(d), self.n - 1)
                nxt = f.select(self.node_axis(d), 0).roll(-1, ea)
                mean = 0.5 * (hi + nxt)
                g.append(self.gradient(f, d, (mean, mean.roll(1, ea))))
            grad.append(g)
        div = sum(grad[d][d] for d in range(dim))
        kappa = GAMMA / ((GAMMA - 1.0) * PRANDTL)
        out = []
        for d in range(dim):
            tau = [grad[c][d] + grad[d][c] - (2.0 / 3.0 * div if c == d else 0.0)
                   for c in range(dim)]
            heat = kappa * grad[d][dim]
            energy = sum(v[c] * tau[c] for c in range(dim)) + heat
            out.append([torch.zeros_like(p)] + [-MU * t for t in tau] + [-MU * energy])
        return out

    def double_mach(self, x, y, t):
        post = x < 1.0 / 6.0 + (y + 20.0 * t) / math.sqrt(3.0)
        out = []
        for a, b in zip(self._conserved(8.0, 8.25 * math.cos(math.pi / 6.0),
                                        -8.25 * math.sin(math.pi / 6.0), 116.5),
                        self._conserved(1.4, 0.0, 0.0, 1.0)):
            out.append(torch.where(post, torch.full_like(x + y, a), torch.full_like(x + y, b)))
        return out

    @staticmethod
    def _conserved(rho, v1, v2, p):
        return rho, rho * v1, rho * v2, p / (GAMMA - 1.0) + 0.5 * rho * (v1 * v1 + v2 * v2)

    def boundaries(self, s, t, d, hi, lo):
        """Overwrites the outer faces of the double Mach reflection domain."""
        n, u = self.n, s[0]
        x, y = _axes(self.case, self.dev)
        if d == 0:  # faces (ny, nx, j)
            first = [f[:, 0, :, 0] for f in u]
            state = self.double_mach(x[:, 0, :, 0], y[:, 0, :, 0], t)
            f = self.surface_flux(self.prim(state), self.prim(first), 0)
            last = [g[:, -1, :, n - 1] for g in u]
            mean = [g[:, -1].mean(-1) for g in u]
            h = self.surface_flux(self.prim(last), self.prim(mean), 0)
            for q in range(4):
                lo[q][:, 0], hi[q][:, -1] = f[q], h[q]
        else:  # faces (ny, nx, i)
            first = [f[0, :, 0, :] for f in u]
            xf = x[0, :, 0, :]
            state = self.double_mach(xf, y[0, :, 0, :], t)
            wall = [first[0], first[1], -first[2], first[3]]
            outer = [torch.where(xf < 1.0 / 6.0, a.expand_as(b), b) for a, b in zip(state, wall)]
            f = self.surface_flux(self.prim(outer), self.prim(first), 1)
            last = [g[-1, :, n - 1, :] for g in u]
            state = [g.expand_as(last[0]) for g in
                     self.double_mach(xf, y[-1, :, n - 1, :], t)]
            h = self.surface_flux(self.prim(last), self.prim(state), 1)
            for q in range(4):
                lo[q][0], hi[q][-1] = f[q], h[q]

    def rhs(self, u_in, t):
        u = self.split(u_in)
        s = self.prim(u)
        n, dim, nv = self.n, self.dim, self.dim + 2
        alpha = self.alpha(u) if self.case["hg"] else None
        w_visc = self.viscous(*s) if self.case["viscous"] else None
        total = [0.0] * nv
        for d in range(dim):
            ax, ea = self.node_axis(d), self.elem_axis(d) + 1
            nodes = [self.at(s, d, m) for m in range(n)]
            acc = [[torch.zeros_like(nodes[0][2]) for _ in range(nv)] for _ in range(n)]
            for m in range(n):
                for k in range(m + 1, n):
                    f = self.volume_flux(nodes[m], nodes[k], d)
                    a, b = 2.0 * float(self.d[m, k]), 2.0 * float(self.d[k, m])
                    for q in range(nv):
                        acc[m][q] = acc[m][q] + a * f[q]
                        acc[k][q] = acc[k][q] + b * f[q]
            if alpha is not None:
                for m in range(n):
                    acc[m] = [(1.0 - alpha) * a for a in acc[m]]
                for m in range(1, n):
                    f = self.llf(nodes[m - 1], nodes[m], d)
                    wl, wr = alpha / float(self.w[m - 1]), alpha / float(self.w[m])
                    for q in range(nv):
                        acc[m - 1][q] = acc[m - 1][q] + wl * f[q]
                        acc[m][q] = acc[m][q] - wr * f[q]
            if w_visc is not None:
                lines = [f.unbind(ax) for f in w_visc[d]]
                for m in range(n):
                    for q in range(nv):
                        acc[m][q] = acc[m][q] + sum(float(self.dhat[m, k]) * lines[q][k]
                                                    for k in range(n))
            shift = lambda f, k: f.roll(k, ea)
            right = ([shift(f, -1) for f in nodes[0][0]], [shift(f, -1) for f in nodes[0][1]],
                     shift(nodes[0][2], -1))
            hi = self.surface_flux(nodes[n - 1], right, d)
            if w_visc is not None:  # one-sided viscous flux of the high-side element
                hi = [f + shift(w.select(ax, 0), -1) for f, w in zip(hi, w_visc[d])]
            lo = [shift(f, 1) for f in hi]
            if self.case["flow"] == "dmr":
                hi = [f.clone() for f in hi]
                self.boundaries(s, t, d, hi, lo)
            for q in range(nv):
                acc[n - 1][q] = acc[n - 1][q] + hi[q] / float(self.w[n - 1])
                acc[0][q] = acc[0][q] - lo[q] / float(self.w[0])
                line = torch.stack([acc[m][q] for m in range(n)], ax)
                total[q] = total[q] - (2.0 / self.h[d]) * line
        return self.join(total)

    def step(self, u, t, dt):
        u1 = u + dt * self.rhs(u, t)
        u2 = 0.75 * u + 0.25 * (u1 + dt * self.rhs(u1, t + dt))
        return u / 3.0 + 2.0 / 3.0 * (u2 + dt * self.rhs(u2, t + 0.5 * dt))

    def kinetic_energy(self, u):
        w = torch.from_numpy(self.w).to(u)
        parts = self.split(u)
        ke = 0.5 * (parts[1] ** 2 + parts[2] ** 2) / parts[0]
        ww = w[:, None] * w[None, :]
        return (ke * ww).sum() / (ww.sum() * math.prod(self.cells))

    def gradient_of_energy(self, u0, dt, steps):
        states = [u0]
        for k in range(steps):
            states.append(self.step(states[-1], k * dt, dt))
        u = states[-1].detach().requires_grad_(True)
        value = self.kinetic_energy(u)
        (lam,) = torch.autograd.grad(value, u)
        for k in reversed(range(steps)):
            u = states[k].detach().requires_grad_(True)
            with torch.enable_grad():
                (lam,) = torch.autograd.grad(self.step(u, k * dt, dt), u, lam)
        return float(value.detach()), lam


def exact(case, seed):
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    if case["op"] == "batch":
        out = []
        for k, m in enumerate(_batch_members(case)):
            u, method, dt = _state(m, 1000 * seed + k, dev), _Method(m, dev), _dt(m)
            for s in range(case["steps"]):
                u = method.step(u, s * dt, dt)
            out.append(u.reshape(-1))
        return torch.cat(out)
    u, method, dt = _state(case, seed, dev), _Method(case, dev), _dt(case)
    if case["op"] == "rhs":
        return method.rhs(u, 0.0)
    if case["op"] == "gradient":
        return method.gradient_of_energy(u, dt, case["steps"])
    for s in range(case["steps"]):
        u = method.step(u, s * dt, dt)
    return u
