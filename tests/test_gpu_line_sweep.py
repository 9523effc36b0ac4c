"""The line shapes (0-2: sweep and split form) where they can go wrong: meshes whose
rows straddle warps and blocks, a single element across (its own neighbour),
partly filled warps at every degree, steep nodal jumps (the general path of
the volume term next to lines that stay on the series), and states that are
not aligned for vector accesses.

Bars: against the oracle the parity bar (RTOL, another summation order of the
same FP64 terms); shapes 0-2 and aligned against unaligned states bit for bit
(the same arithmetic)."""
from __future__ import annotations

import ctypes
import math

import numpy as np
import pytest

from oracle import dgsem_oracle as do
from tests._util import RTOL, dev_to_ref, ref_to_dev, rel_linf
from tests.test_gpu_parity import make_device, make_oracle

pytestmark = pytest.mark.gpu

CASES = []
for n in range(2, 9):
    for cells, vf in (((37, 3), "chandrashekar"), ((1, 5), "ranocha")):
        CASES.append(dict(ndims=2, polydeg=n - 1, cells=cells, left=(-5.0, -5.0),
                          right=(5.0, 5.0), ic="vortex", vf=vf))
for n in range(2, 6):
    for cells, vf in (((9, 2, 3), "chandrashekar"), ((1, 3, 2), "kennedy_gruber")):
        CASES.append(dict(ndims=3, polydeg=n - 1, cells=cells, left=(0.0,) * 3,
                          right=(2 * math.pi,) * 3, ic="tgv3d", vf=vf))


def _state(case, s):
    """Smooth with a steep patch: density and energy jump by up to a factor of
    three between the nodes of every third element."""
    u = do.initial_state(s, case["ic"])
    rng = np.random.default_rng(case["polydeg"])
    jump = np.ones(u.shape[:-1])
    flat = jump.reshape(math.prod(case["cells"]), -1)
    flat[::3] = rng.uniform(1.0, 3.0, flat[::3].shape)
    return u * jump[..., None]


def _ids(case):
    return f"{case['ndims']}d_p{case['polydeg']}_{case['cells'][0]}_{case['vf']}"


@pytest.mark.parametrize("case", CASES, ids=_ids)
def test_line_sweeps_steep_and_ragged(case, cuda):
    import torch
    vf = case["vf"]
    kw = {k: v for k, v in case.items() if k != "vf"}
    s = make_oracle(kw, volume_flux=vf)
    u_ref = _state(case, s)
    ref = do.rhs(s, u_ref, 0.0)
    solver = make_device(kw, volume_flux=vf)
    u = torch.from_numpy(ref_to_dev(u_ref, case["ndims"])).to(cuda)
    outs = []
    for v in range(3):
        solver.set_launch_variant(v)
        du = torch.empty_like(u)
        solver.rhs(u, du, 0.0)
        outs.append(du)
    torch.cuda.synchronize()
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
    got = dev_to_ref(outs[0].cpu().numpy(), solver.mesh.n_cells)
    assert rel_linf(got, ref) <= RTOL, rel_linf(got, ref)


@pytest.mark.parametrize("ndims,polydeg", [(2, 1), (2, 3), (2, 5), (2, 7), (3, 1), (3, 2), (3, 3)])
def test_line_sweeps_unaligned_states(ndims, polydeg, cuda):
    """u_n, u_in and u_out of a stage at an odd multiple of 8 bytes."""
    import torch

    from dgsem_b200 import _capi as C
    cells = (7, 3) if ndims == 2 else (5, 2, 3)
    case = dict(ndims=ndims, polydeg=polydeg, cells=cells, left=(0.0,) * ndims,
                right=(2 * math.pi,) * ndims, ic="tgv2d" if ndims == 2 else "tgv3d")
    s = make_oracle(case)
    u = torch.from_numpy(ref_to_dev(do.initial_state(s, case["ic"]), ndims)).to(cuda)
    v = 1.001 * u
    solver = make_device(case)

    def stage(u_n, u_in, out):
        C.check(C.lib().dgsem_ssprk3_stage(
            solver.handle, 2, ctypes.c_void_p(u_n.data_ptr()), ctypes.c_void_p(u_in.data_ptr()),
            ctypes.c_void_p(out.data_ptr()), 0.0, 1.0e-3), "stage")
        torch.cuda.synchronize()
        return out

    def shifted(t):
        buf = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)
        buf[1:].copy_(t.reshape(-1))
        return buf[1:]

    for shape in range(3):
        solver.set_launch_variant(shape)
        want = stage(u, v, torch.empty_like(u))
        got = stage(shifted(u), shifted(v), shifted(torch.zeros_like(u)))
        assert torch.equal(want.reshape(-1), got), shape
