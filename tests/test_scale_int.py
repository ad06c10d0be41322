"""CPU check that the channels' integer scaling (csrc/scale_int.cuh) gives the
FP64 product bit for bit.  Compiled with g++, no GPU."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_scale_int_is_the_fp64_product(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    exe = tmp_path / "scale_int_check"
    res = subprocess.run(["g++", "-O2", "-std=gnu++17", "-I" + os.path.join(ROOT, "quantumlab_gb300", "csrc"),
                          os.path.join(ROOT, "tests", "native", "scale_int_check.cpp"), "-o", str(exe)],
                         capture_output=True, text=True)
    assert res.returncode == 0, res.stderr
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    v = {k: int(x) for k, x in (line.split() for line in out.stdout.strip().splitlines())}
    assert v["wrong"] == 0 and v["products"] > 5e6, v
