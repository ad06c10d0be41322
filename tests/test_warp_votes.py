"""Warp votes name the lanes that take part (csrc/*.cu).  __activemask() tells
which lanes happen to run together; it does not make them meet at the vote.  A
check of the sources, no GPU."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "quantumlab_gb300", "csrc")


def test_no_vote_over_the_active_mask():
    for path in glob.glob(os.path.join(CSRC, "*.cu*")):
        assert "__activemask" not in re.sub(r"//[^\n]*", "", open(path).read()), path
