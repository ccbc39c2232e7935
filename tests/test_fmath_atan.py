"""CPU: the gradient's atan2 (slm_atan2f_cr, csrc/fmath_cr.h) against the double
function rounded to float, compiled for the host from the source the kernels
use, with each reciprocal exact and one ulp to either side (the device takes an
approximate one; the result must not depend on it)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "skylens-stream-rs_gb300", "csrc")


@pytest.mark.parametrize("ulp", [0, 1, -1])
def test_atan2f_equals_double_rounded(tmp_path, ulp):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no g++")
    exe = str(tmp_path / "check")
    subprocess.check_call([gxx, "-O2", "-std=c++17", "-ffp-contract=off", f"-DSLM_FM_RCP_ULP={ulp}", "-I", CSRC, "-o", exe,
                           os.path.join(HERE, "fmath_atan_check.cpp"), "-lm"])
    r = subprocess.run([exe, "4000000"], capture_output=True, text=True, timeout=600)
    bad, n = map(int, r.stdout.split()[-2:])
    assert bad == 0 and n > 4_000_000, r.stdout
