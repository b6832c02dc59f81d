"""The screened predecessor search of the DTW kernel (csrc/dtw_row.cuh), built
for the host: every decision equals the unscreened program's, and the division
by a fixed divisor equals the division."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.skipif(shutil.which("g++") is None, reason="no C++ compiler")
def test_screened_decisions_equal_the_program(tmp_path):
    exe = str(tmp_path / "dtw_row_host")
    subprocess.run(["g++", "-O2", "-std=c++17", "-mfma", "-ffp-contract=off", "-Wno-unknown-pragmas",
                    os.path.join(HERE, "dtw_row_host.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe, "4"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout
