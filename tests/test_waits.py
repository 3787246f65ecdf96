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


@pytest.mark.parametrize("path", [p for p in SOURCES if os.path.basename(p) not in ("common.cuh", "qwen35_ops.cu", "recurrent_mixers.cu")], ids=os.path.basename)
def test_run_outs_are_counted_behind_every_role(path):
    """A thread that counts at the end of its own role misses what runs out in the others after that: behind the count's place no wait may follow, and a
    barrier of all roles lies before it (a role that returns early arrives there)."""
    text = open(path).read()
    waits = [m.start() for m in re.finditer(r"mbar_wait_bounded\(", text)]
    counts = [m.start() for m in re.finditer(r"count_run_out\(", text)]
    assert len(counts) == (1 if waits else 0)
    if waits and os.path.basename(path) != "runtime.cu":  # (one thread there)
        assert max(waits) < counts[0]
        gap = text[max(waits):counts[0]]
        assert "__syncthreads();" in gap or 'bar.sync 2, %0;" ::"n"(kDcThreads)' in gap
        for m in re.finditer(r"\n    return;\n", text[min(waits):counts[0]]):
            before = text[min(waits):counts[0]][:m.start()]
            assert before.endswith('asm volatile("bar.arrive 2, %0;" ::"n"(kDcThreads) : "memory");')


REFUSAL = """
import torch
from pegainfer_b200 import ffi
from pegainfer_b200.config import QWEN3_TINY
from pegainfer_b200.model import ModelRuntimeConfig, Qwen3Model
from pegainfer_b200.qwen35 import QWEN35_TINY, Qwen35Model, iter_random_weights
from pegainfer_b200.synthetic import random_weights
from tests.test_vegodra_gpu import build, cfg_edges, make_weights

lib = ffi.lib()
assert lib.pk_b200_wait_errors() == -1 and lib.pk_b200_wait_errors_seen() == 0  # nothing is counted before the first cublas_init
w3 = {k: v.cuda() for k, v in random_weights(QWEN3_TINY, seed=0).items()}
w35 = {k: v.cuda() for k, v in iter_random_weights(QWEN35_TINY, seed=0)}
cfg = cfg_edges()
wv = make_weights(cfg, 1)


def make():
    a, b, c = Qwen3Model(QWEN3_TINY, w3, ModelRuntimeConfig(num_pages=16)), Qwen35Model(QWEN35_TINY, w35, num_pages=16), build(cfg, wv, torch.bfloat16)
    kv, r35, rv = a.alloc_kv(), b.alloc_request(), c.alloc_request()
    return (a, b, c), [("qwen3 prefill", lambda: a.prefill([[1, 2, 3]], [kv])), ("qwen3 decode", lambda: a.decode([4], [kv])),
                       ("qwen3.5 prefill", lambda: b.prefill(r35, [1, 2, 3])), ("qwen3.5 decode", lambda: b.decode(r35, 4)),
                       ("layer list", lambda: c.step([(rv, [1, 2, 3])]))]


old, steps = make()
for _, s in steps:
    s()
assert lib.pk_b200_wait_errors() == 0
assert lib.pk_b200_wait_probe(0, None) == -1 and lib.pk_b200_wait_probe(4, None) == 0
assert lib.pk_b200_wait_errors() == 1 and lib.pk_b200_wait_errors_seen() == 1
for what, s in steps:
    try:
        s()
    except RuntimeError as e:
        assert "gave up a wait" in str(e), (what, str(e))
    else:
        raise AssertionError(what + " was not refused")
new, steps = make()  # models made afterwards work
for _, s in steps:
    s()
torch.cuda.synchronize()  # and the device does
for m in old + new:
    m.close()
print("refused and served")
"""


@pytest.mark.gpu
def test_steps_behind_a_run_out_wait_are_refused():
    """in a process of its own: the count stays"""
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(CSRC))
    run = subprocess.run([sys.executable, "-c", REFUSAL], cwd=root, env=dict(os.environ, PYTHONPATH=root), capture_output=True, text=True, timeout=300)
    assert run.returncode == 0 and "refused and served" in run.stdout, run.stdout[-2000:] + run.stderr[-4000:]
