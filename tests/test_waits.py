"""Waits with a limit (mbar_wait_bounded, csrc/common.cuh): what a kernel does once one of them has run out.  No GPU is made to hang for it: the
protocol is checked in the sources, and on a GPU a barrier that nothing completes is waited for with a short limit."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pegainfer_b200", "csrc")
SOURCES = sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")))


def block_after(text, at):
    """the brace-enclosed block that opens at or behind `at`"""
    i = text.index("{", at)
    depth = 0
    for j in range(i, len(text)):
        depth += {"{": 1, "}": -1}.get(text[j], 0)
        if depth == 0:
            return text[i:j + 1]
    raise AssertionError("unbalanced braces")


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_no_loop_with_a_barrier_ends_on_a_threads_own_view_of_the_flag(path):
    """A loop over a barrier of several warps must end for all of them alike: a warp that sees the flag before another leaves that one waiting for good."""
    text = open(path).read()
    for m in re.finditer(r"\b(?:for|while) \([^{}]*\*dead[^{}]*\) \{", text):
        body = block_after(text, m.end() - 1)
        assert not re.search(r"bar\.sync|__syncthreads|barrier\.cluster", body), f"{os.path.basename(path)}: {m.group(0)}"
