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


LOST_PEER = """
import ctypes as C
import torch
from pegainfer_b200 import ffi

lib = ffi.lib()
lib.cuda_set_device(0)
lib.cublas_init()
assert lib.pk_tp_set_wait_limit(None, 5) == -1


def comm():  # a rank of two whose peer never comes
    stage = [torch.zeros(1 << 20, dtype=torch.uint8, device="cuda") for _ in range(2)]
    flags = [torch.zeros(int(lib.pk_tp_flag_bytes()), dtype=torch.uint8, device="cuda") for _ in range(2)]
    c = lib.pk_tp_comm_create(0, 2, (C.c_void_p * 2)(*[s.data_ptr() for s in stage]), (C.c_void_p * 2)(*[f.data_ptr() for f in flags]), 1 << 20)
    assert lib.pk_tp_set_wait_limit(c, 0) == -1 and lib.pk_tp_set_wait_limit(c, 5000) == 0
    return c, stage, flags


bf = lambda *s: torch.ones(*s, device="cuda").bfloat16()
x, w, y, h, hidden = bf(1, 1024), bf(512, 1024), bf(1, 512), bf(4, 512), bf(1, 1024)
step, idx = torch.zeros(1, dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")


def gemv(c, x_mode, epi):
    g = ffi.GemvArgs()
    g.W, g.X, g.residual, g.norm_w = w.data_ptr(), x.data_ptr(), x.data_ptr(), x.data_ptr()
    g.Y = (C.c_void_p * 3)(y.data_ptr(), None, None)
    g.seg_rows = (C.c_int * 3)(512, 0, 0)
    g.M, g.N, g.K, g.x_mode, g.epi, g.eps = 512, 1, 1024, x_mode, epi, 1e-6
    g.hidden_out = hidden.data_ptr() if x_mode else None
    g.tp_comm, g.tp_step, g.tp_op = c, step.data_ptr(), 0
    return lib.pk_b200_gemv_fused(C.byref(g), None)


calls = [lambda c: lib.pk_tp_all_reduce_rows(c, h.data_ptr(), 512, 4, None), lambda c: lib.pk_tp_top1_exchange(c, y.data_ptr(), idx.data_ptr(), 1, 0, None, 9, None),
         lambda c: gemv(c, 0, 3), lambda c: gemv(c, 2, 0)]
keep = []
for n, call in enumerate(calls):
    keep.append(comm())
    if n == 3:  # x_mode 2 waits for the number that its own flags name
        keep[-1][2][0].view(torch.int32)[2 * 64 * 8] = 1
    torch.cuda.synchronize()
    for _ in range(2):  # the second call's waits give up at once, and are not counted again
        assert call(keep[-1][0]) == 0 and lib.pk_b200_wait_errors() == n + 1, n
assert torch.equal(x + x, 2 * x)  # the context works
print("counted and returned")
"""


@pytest.mark.gpu
def test_a_peer_that_never_comes_is_counted():
    """in a process of its own: the count stays"""
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(CSRC))
    run = subprocess.run([sys.executable, "-c", LOST_PEER], cwd=root, env=dict(os.environ, PYTHONPATH=root), capture_output=True, text=True, timeout=300)
    assert run.returncode == 0 and "counted and returned" in run.stdout, run.stdout[-2000:] + run.stderr[-4000:]
