"""The rule by which a lane stays in fixed point (fx_math.cuh), on the host: a
lane that stays has no output part that depends on small parts alone."""
import os
import shutil
import subprocess

import pytest

from tests.test_plan_host import ROOT, _cuda_include


def test_lanes_that_stay(tmp_path):
    cxx, inc = shutil.which("g++"), _cuda_include()
    if not cxx or not inc:
        pytest.skip("needs g++ and the CUDA headers")
    exe = tmp_path / "fx_rule_check"
    subprocess.run([cxx, "-std=c++17", "-O1", "-I", os.path.join(ROOT, "include"),
                    "-I", os.path.join(ROOT, "kfft_gb300", "csrc"), "-I", inc,
                    os.path.join(ROOT, "tests", "fx_rule_check.cpp"), "-o", str(exe)],
                   check=True, capture_output=True, text=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=120).stdout
    stay, leave, wrong, exact_lost = map(int, out.split())
    assert stay > 10000 and leave > 5000
    assert wrong == 0
    assert exact_lost == 0
