"""The cluster's plan of an LP whose vectors do not fit beside each other (sih26_b200/csrc/resident_plan.cuh) on
the CPU: never taken for one that fits (an LP without rows or columns neither), in turns while either vector fits
the shared memory alone, else without any."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CUDA_INC = "/usr/local/cuda/include"


def test_outside_plans(tmp_path):
    if shutil.which("g++") is None or not os.path.isdir(CUDA_INC):
        pytest.skip("no C++ compiler or CUDA headers")
    exe = tmp_path / "plan_check"
    r = subprocess.run(["g++", "-O1", "-std=c++17", "-w", "-I", CUDA_INC, "-I", os.path.join(ROOT, "include"),
                        "-I", os.path.join(ROOT, "sih26_b200", "csrc"), os.path.join(HERE, "plan_check.cpp"),
                        "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    smem = 212 * 1024
    whole = smem // 8
    sizes = [(0, 6000), (6000, 0), (0, 2 * whole), (2 * whole, 0), (whole, whole), (1, whole + 1), (whole + 1, 1)]
    out = subprocess.run([str(exe), *(str(v) for s in sizes for v in s)], capture_output=True, text=True)
    got = [tuple(map(int, line.split())) for line in out.stdout.splitlines()]
    assert got == [(8, 1, smem) if max(s) <= whole else (8, 2, 0) for s in sizes]
