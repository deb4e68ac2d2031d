"""The FP64 kernels' quotient whose operands are tested apart from it (mquo
with mout, mpos and mrcpp in csrc/hp_kernels.cuh): whatever is not flagged
equals the hardware IEEE quotient bit for bit, zeros with their sign, and
nothing inside the documented ranges is flagged.  The magnitudes cover the
whole range, its two ends, and the wider range of the least-squares products
(2^[-900, 800)), whose factors are tested instead."""
import os
import re
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = str(tmp_path_factory.mktemp("quotient") / "check")
    subprocess.run([nvcc, "-O3", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-fmad=false",
                    "-o", exe, os.path.join(HERE, "quotient_check.cu")], check=True, capture_output=True)
    return exe


@pytest.mark.parametrize("lo,hi,test", [(-1022, 1024, 0), (-803, -797, 0), (798, 804, 0), (-1022, 1024, 1),
                                        (-803, -797, 1), (798, 804, 1), (-900, 800, 2)])
def test_unflagged_quotients_are_ieee(check, lo, hi, test):
    out = subprocess.run([check, str(lo), str(hi), str(test)], capture_output=True, text=True, timeout=300)
    m = re.search(r"pairs (\d+) flagged (\d+) mismatches (\d+) wrong (\d+)", out.stdout)
    assert m, out.stdout + out.stderr
    pairs, flagged, mismatches, wrong = map(int, m.groups())
    assert pairs > 50_000_000 and flagged < pairs and mismatches == 0 and wrong == 0, out.stdout
