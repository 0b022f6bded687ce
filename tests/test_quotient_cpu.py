"""The cluster kernel's division by a divisor known in advance gives the bits of a / b, on the CPU."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def test_quotient_has_the_bits_of_a_division(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("no C++ compiler")
    exe = tmp_path / "quotient_check"
    # no contraction: the only fused operations are the ones written
    r = subprocess.run(["g++", "-O1", "-std=c++17", "-ffp-contract=off", "-I",
                        os.path.join(ROOT, "sih26_b200", "csrc"), os.path.join(HERE, "quotient_check.cpp"),
                        "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout + out.stderr
