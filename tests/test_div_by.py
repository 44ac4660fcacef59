"""div_by (csrc/device/device.cuh): the factorisation's quotients from a
reciprocal of a few ulp.

Bound: with r = (1 + e) / b, |e| <= k 2^-52, the product a r is off by at most
(k + 1) 2^-52 relative; the correction leaves of that the part that r's own
error and the rounding of the remainder make, (k + 1)(k + 2) 2^-104, and the
last rounding adds half an ulp: 0.5 + (k + 1)(k + 2) 2^-51 ulp at most, for
k = 4 half an ulp and 2^-46.  2^-44 is asked for, and at most one ulp from the
division operator, from which random operands then hardly ever differ (ties
within 2^-44 ulp: none expected of 2^20)."""
import os
import re
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = os.path.join(ROOT, "tests", "cxx", "div_by_test.cu")
INC = "-I" + os.path.join(ROOT, "hfls_b200", "csrc", "device")


def run(cmd, exe):
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    rows = re.findall(r"(.+) max_ulp_excess (\S+) differ (\d+) apart (\d+) of (\d+)", r.stdout)
    for what, excess, differ, apart, n in rows:
        assert float(excess) <= 2.0 ** -44 and int(apart) == 0 and int(differ) <= 1, r.stdout
        assert int(n) == 1 << 20
    return len(rows)


def test_reciprocals_up_to_four_ulp_off(tmp_path):
    exe = str(tmp_path / "div_by")
    assert run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-x", "c++", INC, SRC, "-o", exe], exe) == 9


@pytest.mark.gpu
def test_reciprocals_of_the_kernels(tmp_path):
    nvcc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    exe = str(tmp_path / "div_by")
    assert run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O2", INC, SRC, "-o", exe], exe) == 2
