"""The two forms of the line shapes (0-2) with every scheme they carry: split
(a block per group of elements) on small meshes, sweep (a warp per group) on
meshes just above the size at which shape 0 changes over, so that the kernel
shape 0 launches there is the one production meshes run.  States have nodal
jumps of density and pressure, independent of each other, on both sides of the
ranges of the series of the logarithmic means.

Bars: the oracle at the parity bar (RTOL: another summation order of the same
FP64 terms); shapes 0, 1 and 2 bit for bit (the same arithmetic); the
node-parallel shapes 3 and 4, which share the viscous kernel, at RTOL too."""
from __future__ import annotations

import math

import numpy as np
import pytest

from oracle import dgsem_oracle as do
from tests._util import RTOL, dev_to_ref, ref_to_dev, rel_linf
from tests.test_gpu_parity import SF, VF

pytestmark = pytest.mark.gpu

MU, PR = 2.0e-2, 0.72
SPLIT, SWEEP = "stage_split_kernel", "stage_line_kernel"


def _case(ndims, n, cells, form, vf="chandrashekar", sf="llf", hg=False, viscous=False,
          bc="periodic", walls=(None,) * 4):
    return dict(ndims=ndims, n=n, cells=cells, form=form, vf=vf, sf=sf, hg=hg, viscous=viscous,
                bc=bc, walls=walls)


CHANNEL = (None, None, "noslip", "slip")
BOX = ("slip", "noslip", "noslip", "slip")
CASES = [
    # 2D, split form of the scheme
    _case(2, 2, (199, 149), SWEEP, "ranocha"),
    _case(2, 3, (149, 121), SWEEP, "kennedy_gruber"),
    _case(2, 4, (151, 131), SWEEP, "ranocha"),
    _case(2, 4, (149, 133), SWEEP, "chandrashekar", "hllc"),
    _case(2, 5, (127, 121), SWEEP),
    _case(2, 6, (113, 109), SWEEP),
    _case(2, 7, (101, 97), SWEEP, "ranocha"),
    _case(2, 8, (103, 97), SWEEP),
    # shock capturing, double Mach boundaries
    _case(2, 4, (16, 12), SPLIT, hg=True),
    _case(2, 6, (10, 12), SPLIT, hg=True),
    _case(2, 4, (24, 6), SPLIT, sf="hllc", hg=True, bc="dmr"),
    _case(2, 4, (137, 131), SWEEP, "ranocha", "hllc", hg=True),
    _case(2, 4, (264, 66), SWEEP, sf="hllc", hg=True, bc="dmr"),
    _case(2, 4, (262, 66), SWEEP, hg=True, bc="dmr"),
    _case(2, 5, (10, 12), SPLIT, hg=True),
    _case(2, 5, (97, 79), SWEEP, hg=True),
    _case(2, 8, (61, 59), SWEEP, hg=True),
    # viscous terms, with shock capturing, with walls
    _case(2, 4, (9, 7), SPLIT, viscous=True),
    _case(2, 4, (149, 133), SWEEP, viscous=True),
    _case(2, 3, (12, 10), SPLIT, hg=True, viscous=True),
    _case(2, 5, (83, 61), SWEEP, hg=True, viscous=True),
    _case(2, 2, (8, 6), SPLIT, viscous=True, bc="walls", walls=CHANNEL),
    _case(2, 4, (8, 6), SPLIT, viscous=True, bc="walls", walls=BOX),
    _case(2, 5, (8, 6), SPLIT, viscous=True, bc="walls", walls=CHANNEL),
    _case(2, 4, (1, 7), SPLIT, viscous=True, bc="walls", walls=BOX),
    _case(2, 3, (7, 1), SPLIT, hg=True, viscous=True, bc="walls", walls=BOX),
    _case(2, 4, (149, 133), SWEEP, viscous=True, bc="walls", walls=CHANNEL),
    _case(2, 5, (127, 121), SWEEP, viscous=True, bc="walls", walls=BOX),
    _case(2, 4, (137, 131), SWEEP, hg=True, viscous=True, bc="walls", walls=CHANNEL),
    # 3D
    _case(3, 3, (17, 13, 11), SWEEP, "ranocha"),
    _case(3, 4, (13, 12, 11), SWEEP),
    _case(3, 5, (13, 11, 10), SWEEP),
    _case(3, 2, (4, 3, 3), SPLIT, hg=True),
    _case(3, 3, (4, 3, 3), SPLIT, hg=True),
    _case(3, 4, (4, 3, 3), SPLIT, "ranocha", hg=True),
    _case(3, 5, (4, 3, 3), SPLIT, hg=True),
    _case(3, 4, (13, 12, 11), SWEEP, "kennedy_gruber", hg=True),
    _case(3, 5, (13, 11, 10), SWEEP, hg=True),
    _case(3, 2, (4, 3, 3), SPLIT, viscous=True),
    _case(3, 3, (4, 3, 3), SPLIT, "ranocha", viscous=True),
    _case(3, 5, (3, 3, 2), SPLIT, viscous=True),
    _case(3, 4, (13, 12, 11), SWEEP, viscous=True),
]


def _ids(c):
    tags = [f"{c['ndims']}d_n{c['n']}", c["form"].split("_")[1], c["vf"][:3], c["sf"]]
    tags += [k for k in ("hg", "viscous") if c[k]]
    if c["bc"] != "periodic":
        tags.append(c["bc"] if c["bc"] == "dmr" else "channel" if c["walls"] == CHANNEL else "box")
    return "-".join(tags)


def _domain(c):
    if c["bc"] == "dmr":
        return (0.0, 0.0), (4.0, 1.0)
    return (0.0,) * c["ndims"], (2 * math.pi, math.pi, 5.0)[:c["ndims"]]


def _oracle(c):
    left, right = _domain(c)
    return do.Scheme(ndims=c["ndims"], polydeg=c["n"] - 1, cells=c["cells"], left=left, right=right,
                     periodic=c["bc"] == "periodic", volume_flux=c["vf"], surface_flux=c["sf"],
                     shock_capturing=c["hg"], bc=c["bc"], viscous=c["viscous"], mu=MU, prandtl=PR,
                     walls=c["walls"])


def _solver(c):
    import dgsem_b200 as D
    nd = c["ndims"]
    left, right = _domain(c)
    mesh = D.StructuredMesh(left, right, c["cells"])
    if c["viscous"]:
        eq = (D.CompressibleNavierStokes2D if nd == 2 else D.CompressibleNavierStokes3D)(1.4, MU, PR)
    else:
        eq = (D.CompressibleEuler2D if nd == 2 else D.CompressibleEuler3D)(1.4)
    if c["bc"] == "dmr":
        bcs = [D.DirichletBC("double_mach"), D.OutflowBC(), D.MixedDirichletSlipWallBC("double_mach"),
               D.DirichletBC("double_mach")]
    else:
        wall = {None: D.PeriodicBC, "noslip": D.NSNoSlipAdiabaticWallBC,
                "slip": D.NSSlipAdiabaticWallBC}
        bcs = [wall[k]() for k in (c["walls"] + (None,) * 2)[:2 * nd]]
    vi = D.VolumeIntegralShockCapturingHG if c["hg"] else D.VolumeIntegralSplitForm
    solver = D.StructuredSolver(eq, D.LobattoLegendreBasis(c["n"] - 1), vi(getattr(D, VF[c["vf"]])),
                                getattr(D, SF[c["sf"]])(), mesh, D.BoundarySet(*bcs))
    if c["hg"]:
        solver.set_indicator_parameters(0.5, 0.001, False)
    return solver


def _state(c, s):
    """A smooth flow with nodal jumps in turn over the elements: none, up to a
    ratio of 1.5 in density or pressure or both, up to a ratio of 4."""
    rng = np.random.default_rng(c["n"])
    x = s.geo.coords
    nd = c["ndims"]
    elems = math.prod(c["cells"])
    nodes = x.shape[-2]
    kind = np.arange(elems) % 7
    top = {1: (1.5, 1.0), 2: (1.0, 1.5), 3: (1.5, 1.5), 4: (4.0, 1.0), 5: (1.0, 4.0), 6: (4.0, 4.0)}

    def jumps(k):
        hi = np.array([1.0] + [top[j][k] for j in range(1, 7)])[kind]
        return rng.uniform(1.0, hi[:, None], (elems, nodes)).reshape(x.shape[:-1])

    rho = (1.0 + 0.001 * np.sin(x[..., 0]) * np.cos(2 * x[..., 1])) * jumps(0)
    p = (2.0 + 0.001 * np.cos(x[..., 0] + x[..., 1])) * jumps(1)
    v = [0.4 * np.sin(x[..., 0]) * np.cos(x[..., 1]) + 0.1, -0.3 * np.cos(x[..., 0]) + 0.05,
         0.2 * np.sin(x[..., -1])][:nd]
    return np.stack([rho] + [rho * a for a in v]
                    + [p / 0.4 + 0.5 * rho * sum(a * a for a in v)], axis=-1)


def _forms_of_the_means(c, u):
    """The forms (0 short series, 1 long series, 2 logarithm) that the x lines'
    density mean and inverse mean need."""
    n = c["n"]
    lines = u.reshape(-1, n, u.shape[-1])
    rho = lines[..., 0]
    p = 0.4 * (lines[..., -1] - 0.5 * sum(lines[..., 1 + d] ** 2 for d in range(c["ndims"])) / rho)
    out = []
    for a in (rho, rho / p):
        f2 = ((a[:, :, None] - a[:, None, :]) / (a[:, :, None] + a[:, None, :])) ** 2
        worst = f2.max(axis=(1, 2))
        out.append({int(k) for k in np.digitize(worst, [1.0e-4, 1.0 / 16.0])})
    return out


@pytest.mark.parametrize("case", CASES, ids=_ids)
def test_forms_agree_and_match_oracle(case, cuda):
    import torch
    s = _oracle(case)
    u_ref = _state(case, s)
    if case["vf"] != "kennedy_gruber":
        assert _forms_of_the_means(case, u_ref) == [{0, 1, 2}, {0, 1, 2}]
    t = 0.02
    ref = do.rhs(s, u_ref, t)
    solver = _solver(case)
    u = torch.from_numpy(ref_to_dev(u_ref, case["ndims"])).to(cuda)
    assert solver.kernel_name() == case["form"]
    outs = []
    for shape in range(5):
        solver.set_launch_variant(shape)
        du = torch.empty_like(u)
        solver.rhs(u, du, t)
        solver.check_finite()
        err = rel_linf(dev_to_ref(du.cpu().numpy(), case["cells"]), ref)
        assert err <= RTOL, (shape, solver.kernel_name(), err)
        outs.append(du)
    solver.set_launch_variant(1)
    assert solver.kernel_name() == SPLIT
    solver.set_launch_variant(2)
    assert solver.kernel_name() == SWEEP
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])


@pytest.mark.parametrize("case", [
    _case(2, 4, (8, 6), SPLIT, viscous=True, bc="walls", walls=CHANNEL),
    _case(2, 4, (16, 12), SPLIT, hg=True, viscous=True),
    _case(3, 3, (4, 3, 3), SPLIT, viscous=True),
    _case(3, 3, (4, 3, 3), SPLIT, hg=True)], ids=_ids)
def test_steps_match_oracle(case, cuda):
    import ctypes

    import torch

    from dgsem_b200 import _capi as C
    s = _oracle(case)
    u_ref = _state(case, s)
    dt = 1.0e-4
    want = u_ref
    for k in range(3):
        want = do.ssprk3_step(s, want, k * dt, dt)
    for shape in range(5):
        solver = _solver(case)
        solver.set_launch_variant(shape)
        u = torch.from_numpy(ref_to_dev(u_ref, case["ndims"])).to(cuda)
        C.check(C.lib().dgsem_ssprk3_steps(solver.handle, ctypes.c_void_p(u.data_ptr()), 0.0, dt, 3),
                "steps")
        solver.check_finite()
        got = dev_to_ref(u.cpu().numpy(), case["cells"])
        assert rel_linf(got, want) <= RTOL, shape
        assert rel_linf(got - u_ref, want - u_ref) <= 1e-10, shape


def test_batch_group_above_the_changeover(cuda):
    """A degree group whose meshes together exceed the changeover runs the
    sweep, another in the same batch the split form; each mesh as on its own."""
    import torch

    import dgsem_b200 as D
    specs = [((97, 61), 3), ((83, 79), 3), ((90, 85), 3), ((9, 5), 5), ((7, 11), 5)]
    left, right = (0.0, 0.0), (2 * math.pi, math.pi)
    batch = D.BatchSolver(D.CompressibleEuler2D(1.4),
                          [(D.StructuredMesh(left, right, c), p) for c, p in specs])
    assert [batch.kernel_name(g) for g in range(2)] == [SWEEP, SPLIT]
    parts, dts, want = [], [], []
    for cells, p in specs:
        case = _case(2, p + 1, cells, SPLIT)
        u = torch.from_numpy(ref_to_dev(_state(case, _oracle(case)), 2)).to(cuda)
        solver = _solver(case)
        sol = D.Solution(solver.mesh, solver.basis, solver.eq)
        sol.u.copy_(u)
        D.SSPRK3(sol, solver.mesh, 1e-4).step(solver, sol, 1e-4)
        parts.append(u.reshape(-1))
        want.append(sol.u.reshape(-1).clone())
        dts.append(1e-4)
    want = torch.cat(want)
    for shape in (None, 0, 1, 2):
        if shape is not None:
            batch.set_launch_variant(shape)
        batch.u.copy_(torch.cat(parts))
        batch.step(0.0, dts)
        torch.cuda.synchronize()
        assert torch.equal(batch.u, want), shape
