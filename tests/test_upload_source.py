"""Uploads that are queued and not waited for keep their host memory
(csrc/upload_source.h).  No GPU: the class against a runtime that copies as
late as it may, and the files that queue such uploads."""
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "quantumlab_gb300", "csrc")
CUDA = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")


def test_late_copies_find_their_source(tmp_path):
    if shutil.which("g++") is None or not os.path.exists(os.path.join(CUDA, "cuda_runtime.h")):
        pytest.skip("g++ or the CUDA headers not available")
    exe = tmp_path / "upload_source_check"
    res = subprocess.run(["g++", "-O1", "-std=gnu++17", "-I" + CSRC, "-I" + os.path.join(ROOT, "include"), "-I" + CUDA,
                          os.path.join(ROOT, "tests", "native", "upload_source_check.cpp"), "-o", str(exe)],
                         capture_output=True, text=True)
    assert res.returncode == 0, res.stderr
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0, out.stderr
    v = dict(line.split() for line in out.stdout.strip().splitlines())
    assert int(v["wrong"]) == 0 and int(v["checked"]) > 20000


@pytest.mark.parametrize("name", ["fused_build.cu", "fused_small.cu"])
def test_plan_uploads_go_through_it(name):
    text = open(os.path.join(CSRC, name)).read()
    assert "UploadSource" in text or "scratch.source" in text
    assert not re.search(r"cudaMemcpy\w*\([^;]*HostToDevice", text)
