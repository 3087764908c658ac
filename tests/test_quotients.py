"""The device code's batched FP64 quotients (e4c_quotients.cuh) against IEEE
division, on the CPU: tests/quotients_check.cpp includes the kernels' own file
and compares bits over random operands of the accepted range and beyond it,
mantissas at the ends of the binade, quotients as near to rounding midpoints as a
divisor allows, van Albada operands and zeros of both signs."""
import os
import shutil
import subprocess
import tempfile

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "eilmer4_b200", "csrc")


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_batched_quotients_match_ieee_division():
    with tempfile.TemporaryDirectory() as tmp:
        exe = os.path.join(tmp, "quotients_check")
        subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", CSRC, "-o", exe,
                        os.path.join(HERE, "quotients_check.cpp"), "-lm"], check=True)
        out = subprocess.run([exe, "20000000"], capture_output=True, text=True)
        assert out.returncode == 0, out.stdout + out.stderr
        assert "mismatches 0 0 0" in out.stdout
