"""con2prim's root finder (grhd::root_safe_newton in physics.cuh) skips FP64 residuals whose
outcome an FP32 estimate settles; its iterates and root must stay those of the reference's
iteration (equations.f90:249-340) to the bit.

tests/root_probe.cu includes the shipped header and compares both on 4.2e7 seeded states:
physical ones, ones with no physical state behind them, ones at the edges of the estimate's
range, zero, negative and infinite input, and negative total energy.
"""
import os
import re
import subprocess
import tempfile

import pytest

from grhd_b200 import build

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(HERE, "root_probe.cu")
INC = os.path.join(os.path.dirname(HERE), "grhd_b200", "csrc", "gpu")


def test_screened_root_is_the_reference_root():
    with tempfile.TemporaryDirectory() as d:
        exe = os.path.join(d, "root_probe")
        subprocess.run([build._nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "--fmad=false",
                        "-I", INC, "-o", exe, SRC], check=True, capture_output=True, text=True)
        out = subprocess.run([exe], check=True, capture_output=True, text=True, timeout=120).stdout
    rows = re.findall(r"kind (\d) samples (\d+) bad (\d+)", out)
    assert len(rows) == 5, out
    assert all(int(bad) == 0 for _, _, bad in rows), out
