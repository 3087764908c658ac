"""The device code's batched FP64 quotients (rcp_q, quot in e4c_physics.cuh)
against IEEE division, on the CPU: tests/quotients_check.c restates them in C
and checks random operands over the accepted range, mantissas at the ends of
the binade, quotients as near to rounding midpoints as a divisor allows and van
Albada operands."""
import os
import shutil
import subprocess
import tempfile

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.skipif(shutil.which("gcc") is None, reason="needs gcc")
def test_batched_quotients_match_ieee_division():
    with tempfile.TemporaryDirectory() as tmp:
        exe = os.path.join(tmp, "quotients_check")
        subprocess.run(["gcc", "-O2", "-ffp-contract=off", "-o", exe,
                        os.path.join(HERE, "quotients_check.c"), "-lm"], check=True)
        out = subprocess.run([exe, "20000000"], capture_output=True, text=True)
        assert out.returncode == 0, out.stdout + out.stderr
        assert "mismatches 0 0" in out.stdout
