"""Tensor-core plans without a GPU: the scoring kernel's arithmetic on raw bytes,
with the plan's per-output constants and rotated rows, restated
(tests/native/tc_bytes_check.cpp) equals direct evaluation."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_bytes_constants_and_rotations(tmp_path):
    exe = tmp_path / "tc_bytes_check"
    csrc = os.path.join(ROOT, "idash2019_2_gb300", "csrc")
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", csrc, "-o", str(exe),
                    os.path.join(ROOT, "tests", "native", "tc_bytes_check.cpp"), os.path.join(csrc, "plan.cpp")],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-3000:]
    lines = [ln for ln in r.stdout.splitlines() if ln.startswith("trial")]
    assert len(lines) == 24 and all(" ok:" in ln for ln in lines)
