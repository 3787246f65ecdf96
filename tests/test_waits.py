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
    for m in re.finditer(r"\b(?:for|while) \([^{}]*(?:\*dead|wait_failed)[^{}]*\) \{", text):
        body = block_after(text, m.end() - 1)
        assert not re.search(r"bar\.sync|__syncthreads|barrier\.cluster", body), f"{os.path.basename(path)}: {m.group(0)}"


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_a_run_out_wait_is_counted_where_it_runs_out(path):
    """Counting at a kernel's end, by one thread, misses the waits of roles that run out after that thread has looked: only the wait itself counts."""
    text = open(path).read()
    counts = [m.start() for m in re.finditer(r"atomicAdd\([^;]*\berr\b", text)]
    if os.path.basename(path) != "common.cuh":
        assert not counts
    else:
        at = text.index("bool mbar_wait_bounded(")
        assert len(counts) == 1 and block_after(text, at).find(text[counts[0]:counts[0] + 20]) >= 0


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_the_word_that_counts_reaches_every_limited_wait(path):
    """every wait with a limit names the flag and the word (WaitFlag), not a flag alone"""
    text = open(path).read()
    for m in re.finditer(r"mbar_wait_bounded\(", text):
        if os.path.basename(path) == "common.cuh":
            continue
        depth, j = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[j], 0)
            j += 1
        assert re.search(r", wf\b[^,]*$", text[m.end():j - 1]), text[m.start():j]
