"""Registers of the plain step kernel (CPU: compiles it, runs nothing).

Four CTAs an SM need at most 128 registers a thread.  The fast run-mode kernel fits
without spills because a branch keeps the two copies of its row apart in the schedule;
a compiler that merges them again shows here.
"""

from __future__ import annotations

import re
import subprocess

import pytest

from conftest import PKG_ROOT

SOURCE = """
#include "swe_step.cuh"
#include "swe_step_pair.cuh"
template __global__ void swe::step_kernel_pair<swe::FastMath, 128, true, false>(const swe::StepLaunch);
template __global__ void swe::step_kernel_pair<swe::FastMath, 128, true, true>(const swe::StepLaunch);
"""


def test_fast_run_kernel_does_not_spill(tmp_path):
    from hybrid_flood_b200 import build

    try:
        nvcc = build.nvcc()
    except RuntimeError:
        pytest.skip("no nvcc")
    src = tmp_path / "step.cu"
    src.write_text(SOURCE)
    r = subprocess.run([nvcc, *build.ARCH_FLAGS, "-O3", "-std=c++17", "--expt-relaxed-constexpr", "-Xptxas", "-v",
                        "-I", str(PKG_ROOT / "csrc"), "-cubin", str(src), "-o", str(tmp_path / "step.cubin")],
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    kernels = re.findall(r"step_kernel_pair.*?(\d+) bytes spill stores, (\d+) bytes spill loads.*?Used (\d+) registers",
                         r.stderr, re.S)
    assert len(kernels) == 2
    for stores, loads, registers in kernels:
        assert (int(stores), int(loads)) == (0, 0) and int(registers) <= 128
