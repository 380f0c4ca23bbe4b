"""Shuffle masks in the kernels name lanes that are known to take part.

__activemask() reports the lanes that execute together at that instant and
promises nothing about lanes that a loop has split off, so it is no mask for a
shuffle: a lane may then read from one outside it.  It stands only inside a
vote, whose result is the same for any split."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "bd_aging_b200", "csrc")


def test_activemask_only_in_votes():
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh")):
            continue
        with open(os.path.join(CSRC, name)) as f:
            code = re.sub(r"//[^\n]*", "", f.read())
        votes = len(re.findall(r"__(?:all|any)_sync\(__activemask\(\)", code))
        assert code.count("__activemask()") == votes, name
