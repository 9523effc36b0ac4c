"""bench.py's roofline figures come from the committed ncu summary of the kernel
that runs: every summary of a benchmark workload belongs to a kernel the library
names and carries the figures bench.py reads, and the kernels that the workloads
run by default have one."""
from __future__ import annotations

import os
import re

import pytest

import bench

PROFILES = os.path.join(bench.ROOT, "profiles")
SUMMARIES = sorted(m.groups() for m in (re.match(r"(stage_\w+_kernel)_([a-z]+\d*)\.md$", f)
                                        for f in os.listdir(PROFILES)) if m)
WORKLOADS = set(bench.WORKLOADS) | {"batched"}


@pytest.mark.parametrize("kernel,workload", [s for s in SUMMARIES if s[1] in WORKLOADS])
def test_summary_names_a_kernel_and_its_traffic(kernel, workload):
    assert kernel in bench.KERNEL_DESCRIPTIONS
    key = "traffic_bytes_per_stage" if workload == "batched" else "traffic_bytes_per_launch"
    assert bench.profile_value(workload, kernel, key) > 0.0


@pytest.mark.parametrize("kernel,workload", [
    ("stage_line_kernel", "tgv16"), ("stage_line_kernel", "tgv32"),
    ("stage_line_kernel", "kh1024"), ("stage_split_kernel", "kh64"),
    ("stage_node_kernel", "dmr"), ("stage_line_kernel", "batched")])
def test_default_kernels_have_a_summary(kernel, workload):
    if workload != "batched":
        assert bench.profile_value(workload, kernel, "fp64_flops_per_dof") > 0.0
    assert (kernel, workload) in SUMMARIES
