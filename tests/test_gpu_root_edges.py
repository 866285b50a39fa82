"""con2prim's root finder at the limits of its FP32 screen: NaN operands (which return at once),
Q2 far above E^2, |D / E| at 1.25, and cells nearly at rest.  The root and the flags of the plain
iteration, bit for bit, on 1.7e7 seeded operands (tests/root_edge_probe.cu)."""
import os
import re
import subprocess
import tempfile

import pytest

from grhd_b200 import build

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(HERE, "root_edge_probe.cu")


def test_screened_root_at_its_limits():
    with tempfile.TemporaryDirectory() as d:
        exe = os.path.join(d, "root_edge_probe")
        subprocess.run([build._nvcc(), *build.ARCH, "-O3", "-std=c++17", "--fmad=false", "-I",
                        os.path.join(build.CSRC, "gpu"), "-o", exe, SRC], check=True, capture_output=True, text=True)
        out = subprocess.run([exe], check=True, capture_output=True, text=True, timeout=120).stdout
    rows = re.findall(r"kind (\d) samples (\d+) bad (\d+)", out)
    assert len(rows) == 4 and all(int(n) == 1 << 22 for _, n, _ in rows), out
    assert all(int(bad) == 0 for _, _, bad in rows), out
