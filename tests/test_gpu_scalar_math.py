"""The branch-free reciprocals, quotient and root of the kernels (csrc/physics.cuh)
against IEEE division and square root in numpy, over random significands and a
wide range of exponents and at the edges of the range, and what the solver does
with the states that leave it."""
from __future__ import annotations

import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

from oracle import dgsem_oracle as do
from tests._util import CASES, RTOL, dev_to_ref, ref_to_dev, rel_linf
from tests.test_gpu_parity import make_device, make_oracle

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
RECIP, QUOTIENT, SQRT, RECIP_ULP = 0, 1, 2, 3


@pytest.fixture(scope="module")
def evaluate(tmp_path_factory, cuda):
    if not os.path.exists(NVCC):
        pytest.skip("nvcc missing")
    so = str(tmp_path_factory.mktemp("scalar") / "scalar_math.so")
    r = subprocess.run([NVCC, "-std=c++17", "-O3", "-gencode", "arch=compute_100a,code=sm_100a",
                        "-Xcompiler", "-fPIC", "-shared",
                        "-I", os.path.join(ROOT, "dgsem_b200", "csrc"),
                        os.path.join(ROOT, "tests", "cpp", "scalar_math.cu"), "-o", so],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    lib = ctypes.CDLL(so)
    dp = ctypes.POINTER(ctypes.c_double)
    lib.scalar_math_eval.argtypes = [ctypes.c_int, dp, dp, dp, ctypes.c_int]

    def run(op, a, b=None):
        a = np.ascontiguousarray(a, dtype=np.float64)
        b = a if b is None else np.ascontiguousarray(b, dtype=np.float64)
        out = np.empty_like(a)
        p = [x.ctypes.data_as(dp) for x in (a, b, out)]
        assert lib.scalar_math_eval(op, *p, a.size) == 0
        return out

    return run


def _numbers(rng, n, lo, hi):
    """Random significands, exponents lo .. hi, and at every exponent the
    significands next to 1 and 2."""
    m = 1.0 + rng.integers(0, 1 << 52, n) / float(1 << 52)
    edge = np.array([1.0, 1.0 + 2.0 ** -52, 1.5, 2.0 - 2.0 ** -51, 2.0 - 2.0 ** -52])
    ex = rng.integers(lo, hi + 1, n)
    every = np.repeat(np.arange(lo, hi + 1), edge.size)
    return np.concatenate([np.ldexp(m, ex), np.ldexp(np.tile(edge, hi + 1 - lo), every)])


def _ulps(got, want):
    return np.abs(got - want) / np.spacing(np.abs(want))


def test_reciprocal_is_correctly_rounded(evaluate):
    a = _numbers(np.random.default_rng(1), 1 << 23, -1021, 1020)
    got, want = evaluate(RECIP, a), 1.0 / a
    # Markstein's theorem leaves out the significand of all ones: one unit there
    ones = np.frexp(a)[0] == 1.0 - 2.0 ** -53
    assert np.array_equal(got[~ones], want[~ones]), int((got != want)[~ones].sum())
    assert _ulps(got[ones], want[ones]).max() <= 1.0
    assert np.array_equal(evaluate(RECIP, -a), -got)
    near = evaluate(RECIP_ULP, a)
    assert _ulps(near, want).max() <= 1.0
    assert np.mean(near != want) <= 1.0e-3


def test_quotient_and_root_are_correctly_rounded(evaluate):
    rng = np.random.default_rng(2)
    a, b = _numbers(rng, 1 << 23, -400, 400), _numbers(rng, 1 << 23, -400, 400)
    b = rng.permutation(b)
    assert np.array_equal(evaluate(QUOTIENT, a, b), a / b)
    assert np.array_equal(evaluate(QUOTIENT, np.zeros(4), b[:4]), np.zeros(4))
    # the residual of a root needs 106 bits below its argument: above 2^-900
    x = _numbers(rng, 1 << 23, -900, 1020)
    assert np.array_equal(evaluate(SQRT, x), np.sqrt(x))


def test_ends_of_the_range(evaluate):
    tiny, inf = np.finfo(np.float64).tiny, np.inf
    out = evaluate(RECIP, [0.0, -0.0, inf, -inf, np.nan, 0.25 * tiny])
    assert np.isnan(out).all(), out
    out = evaluate(RECIP_ULP, [0.0, -0.0, inf, -inf, np.nan, 0.25 * tiny])
    assert np.isnan(out).all(), out
    out = evaluate(QUOTIENT, np.ones(6), [0.0, -0.0, inf, -inf, np.nan, 0.25 * tiny])
    assert np.isnan(out).all(), out
    out = evaluate(SQRT, [0.0, -0.0, 0.25 * tiny, 9.9e-291])
    assert np.array_equal(out, np.zeros(4)), out
    assert np.isnan(evaluate(SQRT, [-1.0, -tiny, np.nan, inf])).all()
    # up to the smallest argument that is not taken as zero, within one unit
    x = np.geomspace(1.0e-290, 2.0 ** -900, 4096)
    assert _ulps(evaluate(SQRT, x), np.sqrt(x)).max() <= 1.0


BAD = {"zero density": (0, 0.0), "infinite density": (0, np.inf), "infinite energy": (3, np.inf),
       "nan momentum": (1, np.nan)}


@pytest.mark.parametrize("bad", list(BAD))
@pytest.mark.parametrize("vf,sf,hg", [("chandrashekar", "llf", False), ("ranocha", "llf", False),
                                      ("kennedy_gruber", "llf", False),
                                      ("chandrashekar", "hllc", True)])
def test_unusable_state_raises_the_flag(vf, sf, hg, bad, cuda):
    """One unusable node makes its own element's result non-finite and raises
    the non-finite flag in every launch shape; elements that are not its
    neighbours keep their bits."""
    import torch

    from dgsem_b200 import _capi as C
    case = dict(CASES["kh_hg"], shock_capturing=hg)
    solver = make_device(case, volume_flux=vf, surface_flux=sf)
    u = torch.from_numpy(ref_to_dev(do.initial_state(make_oracle(case), "kh"), 2)).to(cuda)
    var, value = BAD[bad]
    v = u.clone()
    v[27, var, 5] = value  # element (3, 3) of 8 x 8, an inner node
    far = [e for e in range(64) if abs(e % 8 - 3) + abs(e // 8 - 3) > 1]
    for shape in range(5):
        solver.set_launch_variant(shape)
        good, out = torch.empty_like(u), torch.empty_like(u)
        solver.rhs(u, good, 0.0)
        solver.check_finite()
        solver.rhs(v, out, 0.0)
        with pytest.raises(C.DgsemError):
            solver.check_finite()
        assert not torch.isfinite(out[27]).all(), shape
        assert torch.equal(out[far], good[far]), shape


def test_zero_pressure_is_usable_where_no_flux_divides_by_it(cuda):
    """Kennedy-Gruber with LLF takes p = 0 (root of a zero sound speed)."""
    import torch
    case = CASES["kh"]
    s = make_oracle(case, volume_flux="kennedy_gruber")
    u_ref = do.initial_state(s, "kh")
    u_ref[2, 3, :, 1:] = 0.0  # at rest: pressure and sound speed are exactly zero
    ref = do.rhs(s, u_ref, 0.0)
    assert np.isfinite(ref).all()
    solver = make_device(case, volume_flux="kennedy_gruber")
    u = torch.from_numpy(ref_to_dev(u_ref, 2)).to(cuda)
    du = torch.empty_like(u)
    for shape in range(5):
        solver.set_launch_variant(shape)
        solver.rhs(u, du, 0.0)
        solver.check_finite()
        got = dev_to_ref(du.cpu().numpy(), solver.mesh.n_cells)
        assert rel_linf(got, ref) <= RTOL, (shape, rel_linf(got, ref))
