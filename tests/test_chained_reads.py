"""Chained kernels (csrc/chain_launch.cuh) are resident while the grid before
them still writes: what they read has to come through ordinary loads.  A
non-coherent load (__ldg, or a pointer that is __restrict__, whose loads the
compiler may turn into one or move over the wait) may return what stood there
before.  A check of the sources, no GPU."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "quantumlab_gb300", "csrc")


def kernels():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__", text):
            brace = text.index("{", m.start())
            depth, end = 0, brace
            while True:
                depth += (text[end] == "{") - (text[end] == "}")
                end += 1
                if depth == 0:
                    break
            signature, body = text[m.start():brace], text[brace:end]
            if "chainStart()" in body:
                yield pytest.param(signature, body, id=re.search(r"\b(k[A-Z]\w*)\s*\(", signature).group(1))


@pytest.mark.parametrize("signature,body", list(kernels()))
def test_chained_kernels_read_coherently(signature, body):
    assert "__restrict__" not in signature + body
    assert "__ldg(" not in body and "ld.global.nc" not in body


def test_chained_kernels_are_found():
    assert len(list(kernels())) >= 15
