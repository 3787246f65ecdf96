"""A wait that runs out ends with an error status that the host reads, never with a trap, which would leave the context (and its user's other work) lost."""
import glob
import os

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pegainfer_b200", "csrc")
SOURCES = sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")))


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_no_trap(path):
    text = open(path).read()
    assert "__trap" not in text and "_or_trap" not in text
