"""CPU check of the fixed-point maps that the plain path's gates run on the
integer pipes (quantumlab_gb300/csrc/fix64.cuh), against quadruple precision
and against the FP64 multiply-add chain.  Compiled with g++, no GPU."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_fix64_bounds(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    exe = tmp_path / "fix64_check"
    res = subprocess.run(["g++", "-O2", "-std=gnu++17", "-I" + os.path.join(ROOT, "quantumlab_gb300", "csrc"),
                          os.path.join(ROOT, "tests", "native", "fix64_check.cpp"), "-o", str(exe)],
                         capture_output=True, text=True)
    assert res.returncode == 0, res.stderr
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr
    v = {k: float(x) for k, x in (line.split() for line in out.stdout.strip().splitlines())}
    print(v)
    for name in ("four", "two"):
        assert v[name + "_excess_units"] <= 0                 # half an ulp plus the units of the header's account
        assert v[name + "_accepted"] > 1e6
        assert v[name + "_refused_inputs"] < 0.1 * v[name + "_accepted"]
        for spread in range(5):
            assert v[f"{name}_rms_fixed_{spread}"] <= v[f"{name}_rms_fp64_{spread}"], (name, spread)
    assert v["unfit_maps_taken"] == 0
    assert v["odd_inputs_taken"] == 0
    assert v["edge_rel"] <= 2.0 ** -52
