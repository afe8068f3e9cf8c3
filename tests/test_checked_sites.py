"""The device functions that store beside a fused step's own update, or read the amounts it adds, test their
indices in the bounds-checked build (LBM_IN) as the separate ghost fill and source kernel do.  Read from the
source: no input reaches an index out of range."""
import os
import re

import pytest

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "city-scale-nlos-acoustic-engine-code_b200",
                   "csrc", "kernels.cu")


def bodies(name):
    """Every definition of device function `name`."""
    text = re.sub(r"//[^\n]*", "", open(SRC).read())
    for m in re.finditer(r"void %s\([^;{]*\)\s*\{" % name, text):
        depth, end = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[end], 0)
            end += 1
        yield text[m.end():end]


@pytest.mark.parametrize("name,count", [("ghost_pair", 2), ("ghost_end", 1), ("keep_face_moments", 1), ("add_sources", 2)])
def test_fused_epilogue_is_checked(name, count):
    found = list(bodies(name))
    assert len(found) == count
    for body in found:
        assert "LBM_IN(" in body
