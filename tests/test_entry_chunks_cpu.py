"""Ranges of entries that end next to 2^31 - 1 are walked to their end and no further, on the CPU (such an LP's
values alone take 17 GB)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def test_chunks_cover_the_range(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("no C++ compiler")
    exe = tmp_path / "entry_chunks_check"
    r = subprocess.run(["g++", "-O1", "-ftrapv", "-std=c++17", "-I", os.path.join(ROOT, "sih26_b200", "csrc"),
                        os.path.join(HERE, "entry_chunks_check.cpp"), "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout + out.stderr
