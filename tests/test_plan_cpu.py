"""The cluster's plan of an LP in windows (sih26_b200/csrc/resident_plan.cuh) on the CPU: every entry of x and
y lies in one window, and a side with nothing to gather still gets one pass, which applies its rows' steps."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CUDA_INC = "/usr/local/cuda/include"


def test_every_side_has_a_window(tmp_path):
    if shutil.which("g++") is None or not os.path.isdir(CUDA_INC):
        pytest.skip("no C++ compiler or CUDA headers")
    exe = tmp_path / "plan_check"
    r = subprocess.run(["g++", "-O1", "-std=c++17", "-w", "-I", CUDA_INC, "-I", os.path.join(ROOT, "include"),
                        "-I", os.path.join(ROOT, "sih26_b200", "csrc"), os.path.join(HERE, "plan_check.cpp"),
                        "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    window = int(subprocess.run([str(exe)], capture_output=True, text=True).stdout)
    sizes = [(0, 6000), (6000, 0), (0, 2 * window + 1), (1, 1), (window, window + 1), (2 * window, 1)]
    out = subprocess.run([str(exe), *(str(v) for s in sizes for v in s)], capture_output=True, text=True)
    got = [tuple(map(int, line.split())) for line in out.stdout.splitlines()[1:]]
    assert got == [(1, max(1, -(-n // window)), max(1, -(-m // window))) for m, n in sizes]
