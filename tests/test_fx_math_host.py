"""Host side of the double build's fixed-point arithmetic (fx_math.cuh), built
with the host compiler: table values against long double, the two-limb form,
and the butterflies' constants."""
import os
import shutil
import subprocess

import pytest

from tests.test_plan_host import ROOT, _cuda_include


@pytest.fixture(scope="module")
def printed(tmp_path_factory):
    cxx, inc = shutil.which("g++"), _cuda_include()
    if not cxx or not inc:
        pytest.skip("needs g++ and the CUDA headers")
    exe = tmp_path_factory.mktemp("fx_math") / "fx_math_check"
    subprocess.run([cxx, "-std=c++17", "-O1", "-I", os.path.join(ROOT, "include"),
                    "-I", os.path.join(ROOT, "kfft_gb300", "csrc"), "-I", inc,
                    os.path.join(ROOT, "tests", "fx_math_check.cpp"), "-o", str(exe)],
                   check=True, capture_output=True, text=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=120).stdout
    return [line.split() for line in out.splitlines()]


def test_cosines_and_sines(printed):
    # ten series terms, each a product and a quotient rounded to 2^-62, and
    # long double's own 2^-64 on either side
    rows = [r for r in printed if r[0] == "cossin"]
    assert len(rows) == 13
    for _, n, worst in rows:
        assert float(worst) <= 16, n


def test_limbs(printed):
    assert [r[1] for r in printed if r[0] == "limbs"] in (["0"], ["1"])


def test_constants(printed):
    rows = [r for r in printed if r[0] == "const"]
    assert len(rows) == 2 * (3 + 5 + 6 + 7 + 8 + 9 + 11 + 12 + 13 + 16)
    for r in rows:
        assert float(r[4]) <= 16, r
    # cos 60 = 1 - 1/2 and cos 120 = 0 - 1/2, exactly
    half = str(-(1 << 63))
    assert [r[1:] for r in printed if r[0] == "half"] == [["1", half, "0", half]]
