"""The device and pinned memory that the library keeps between calls, on the CPU: who gets a chunk again, the
bound, what a failed allocation and the release call give back, and that after a device reset a kept address
is neither handed out nor freed (tests/memory_cache_check.cpp over a fake of the CUDA runtime)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CUDA_INC = "/usr/local/cuda/include"


def test_kept_memory_belongs_to_its_context(tmp_path):
    if shutil.which("g++") is None or not os.path.isdir(CUDA_INC):
        pytest.skip("no C++ compiler or CUDA headers")
    exe = tmp_path / "memory_cache_check"
    r = subprocess.run(["g++", "-O1", "-std=c++17", "-w", "-pthread", "-I", CUDA_INC,
                        "-I", os.path.join(ROOT, "sih26_b200", "csrc"),
                        os.path.join(HERE, "memory_cache_check.cpp"), "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout + out.stderr
