"""The coarse levels' division by the diagonal count without a guard
(flub_gb300/csrc/coarse.cuh): equal to IEEE single-precision a / d for every
finite float32 and d = 3, 5, 6 (and a sample for the powers of two), but for
ties between two denormals at d = 6.  Compiled and run on the host."""
import os
import re
import shutil
import subprocess
import tempfile

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.skipif(shutil.which("gcc") is None, reason="gcc not available")
def test_coarse_division_matches_ieee_division():
    with tempfile.TemporaryDirectory() as d:
        exe = os.path.join(d, "coarse_div_check")
        subprocess.run(["gcc", "-O2", "-ffp-contract=off", "-fopenmp", "-o", exe,
                        os.path.join(HERE, "native", "coarse_div_check.c"), "-lm"], check=True)
        out = subprocess.run([exe], capture_output=True, text=True, timeout=2400)
    assert out.returncode == 0, out.stdout + out.stderr
    checked, ties, bad = (int(x) for x in re.findall(r"\d+", out.stdout))
    assert checked > 3 * 0x7f800000 and bad == 0
    assert ties < 6 * (1 << 23)  # all of them below 6 * 2^-126
