"""Launch shapes persisted by DGSEM_TUNING_FILE: a choice stored with the current
kernels is taken without timing, one stored with earlier kernels (the key format
without a revision, or another revision) is timed again."""
from __future__ import annotations

import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CODE = """
import sys; sys.path.insert(0, {root!r})
import torch
import dgsem_b200 as D
from tests._util import CASES, ref_to_dev
from tests.test_gpu_parity import make_device, make_oracle, initial
case = CASES["kh"]
u = torch.from_numpy(ref_to_dev(initial(case, make_oracle(case)), 2)).cuda()
print("chosen", make_device(case).autotune(u)[0])
"""
OLD_KEY = "d2_n4_vf0_sf0_hg0_ns0_e64_cold"


def _choose(path):
    env = dict(os.environ, DGSEM_TUNING_FILE=str(path))
    env.pop("DGSEM_AUTOTUNE_WARM", None)
    r = subprocess.run([sys.executable, "-c", CODE.format(root=ROOT)], env=env, cwd=ROOT,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    return int(r.stdout.split("chosen", 1)[1])


def test_choices_of_other_kernels_are_timed_again(tmp_path, cuda):
    path = tmp_path / "tuning"
    stale = [f"{OLD_KEY} 4", f"r1_{OLD_KEY} 4"]
    path.write_text("\n".join(stale) + "\n")
    first = _choose(path)
    lines = path.read_text().split("\n")[:-1]
    assert lines[:2] == stale and len(lines) == 3, lines
    key, choice = lines[2].split()
    assert key.endswith(OLD_KEY) and key not in (s.split()[0] for s in stale)
    assert int(choice) == first
    # the stored choice is taken as it stands, whatever timing would give
    other = (first + 1) % 5
    path.write_text(f"{key} {other}\n")
    assert _choose(path) == other
    assert path.read_text() == f"{key} {other}\n"
