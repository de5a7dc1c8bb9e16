"""The integer sums of floats (massiveclicks_gb300/csrc/exact_sum.h) that the count
kernels add their public bins with, compiled with g++, against 128-bit sums: exact to the
rounding of the result, which a pair of floats is not."""
import subprocess
import tempfile
from pathlib import Path

from conftest import ROOT


def test_sums_are_exact():
    with tempfile.TemporaryDirectory() as tmp:
        exe = Path(tmp) / "exact_sum_check"
        cmd = ["g++", "-std=c++17", "-O2", "-Wall", "-Werror", f"-I{ROOT / 'massiveclicks_gb300' / 'csrc'}",
               str(ROOT / "tests" / "host_api" / "exact_sum_check.cpp"), "-o", str(exe)]
        res = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
        assert res.returncode == 0, res.stdout
        res = subprocess.run([str(exe)], stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, timeout=120)
        assert res.returncode == 0 and "BAD 0" in res.stdout, res.stdout
