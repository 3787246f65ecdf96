"""Parity at the configurations the benchmark runs.

The model under test is the FULL Qwen3-4B (36 layers, V = 151,936) on the seed-0 CPU-generated random-init
checkpoint -- the same checkpoint bench.py loads -- teacher-forced against the CPU oracle with the parity rule
(every logit within TOL bf16 ulps of the row's max magnitude; arg-max equal unless the oracle's top-1/top-2 gap is
inside the tolerance), plus the free-running first-divergence index (reported).  The reference's counterpart:
HF bf16 greedy on the real model (scripts/generate_test_data.py:41-52) and the real-model batch/sequential test
(pegainfer-qwen3-4b/src/batch_decode.rs:505-606).

* config 1 (128-token prompt + 64 decode steps, non-partition attention): LIVE oracle, full logit rows.
* config 2 (2048-token prefill + 8 decode steps, split-KV in the reference): the oracle run is ~16 TFLOP of fp32 on
  the CPU, so it is a committed fixture (tests/golden/parity_qwen3-4b_p2048_tp1.npz, generator committed beside it;
  the fixture records a CRC of the checkpoint it was computed on and the test checks it first).
Both run the fused B200 path and the reference's op sequence on our kernels (`fused=False`).
Set PK_SKIP_FULLSIZE=1 to skip (e.g. when iterating on one kernel); PK_FULLSIZE_STEPS trims config 1's decode steps.
"""
import os

import numpy as np
import pytest
import torch

from oracle import qwen3_oracle as O
from pegainfer_b200.config import QWEN3_4B
from pegainfer_b200.model import ModelRuntimeConfig, Qwen3Model
from pegainfer_b200.synthetic import random_weights, synthetic_prompt, to_numpy_bits
from tests.golden import parity_fixture as F
from tests.helpers import bits, logits_agree, oracle_cfg

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(os.environ.get("PK_SKIP_FULLSIZE") == "1", reason="PK_SKIP_FULLSIZE=1")]

# bf16 ulps at the row's max |logit| after 36 layers.  Measured on B200:
# fused 7.4 worst over 65 steps of config 1, 5.4 on config 2; compat 5.9 / 5.0 -- rounding-point flips accumulate as
# ~sqrt(layers) (the 2-4 layer configs of test_model_gpu.py sit at <= 2 with a bound of 6).  12 = 1.6 x the worst seen.
TOL_ULP = 12
CFG1_STEPS = int(os.environ.get("PK_FULLSIZE_STEPS", "64"))
LIVE_BUDGET_S = float(os.environ.get("PK_FULLSIZE_LIVE_BUDGET_S", "240"))  # wall-clock budget of the live oracle run


@pytest.fixture(scope="module")
def w4b():
    return random_weights(QWEN3_4B, seed=0, device="cpu")


@pytest.fixture(scope="module")
def cfg1_oracle(w4b):
    """Oracle logits of config 1: prefill(128) + up to CFG1_STEPS teacher-forced decode steps, and its greedy sequence.

    LIVE on the host cores within a wall-clock budget: the decode loop stops early when the budget is spent (a slow or
    oversubscribed host shortens the comparison instead of failing the suite on a timeout); if not even the prefill fits,
    the committed fixture of the same configuration (tests/golden/parity_qwen3-4b_p128_tp1.npz, 8 steps) takes over."""
    import time
    t0 = time.perf_counter()
    O.set_num_threads(os.cpu_count() or 1)
    orc = O.OracleQwen3(oracle_cfg(QWEN3_4B), to_numpy_bits(w4b), num_pages=(128 + CFG1_STEPS) // 16 + 4)
    kv = orc.alloc_kv()
    # probe: one layer-sized GEMM tells how fast this host is before committing to the prefill
    tp = time.perf_counter()
    O.gemm(orc.ranks[0].layers[0]["gate_up"], np.zeros((128, QWEN3_4B.hidden_size), np.uint16))
    probe = time.perf_counter() - tp
    if probe * 36 * 2.2 > LIVE_BUDGET_S:  # the prefill is ~2.2 x this GEMM per layer
        print(f"\n[fullsize] live oracle too slow on this host (probe {probe:.1f} s): using the committed fixture")
        return None
    want = [orc.prefill([synthetic_prompt(128)], [kv])[0]]
    toks = []
    for _ in range(CFG1_STEPS):
        if time.perf_counter() - t0 > LIVE_BUDGET_S:
            break
        toks.append(O.argmax(want[-1]))
        want.append(orc.decode([toks[-1]], [kv])[0])
    assert orc.last_attention_path in (None, "non_partition")
    print(f"\n[fullsize] live oracle: prefill(128) + {len(toks)} decode steps in {time.perf_counter() - t0:.0f} s")
    del orc
    return want, toks


def _model(w, **kw):
    return Qwen3Model(QWEN3_4B, w, ModelRuntimeConfig(max_batch=1, **kw))


def _teacher_forced(m, prompt, tokens):
    kv = m.alloc_kv()
    got = [bits(m.prefill([prompt], [kv])[0])]
    for t in tokens:
        lg, _ = m.decode([t], [kv])
        got.append(bits(lg[0]))
    m.drop_request(kv)
    return got


REF_LIB = os.path.abspath(os.path.join(os.path.dirname(__file__), "..", "oracle", "_ref", "libkernels_ref.so"))
CFG1_VARIANTS = [("fused", dict(fused=True), None), ("compat", dict(fused=False), 16)]
if os.path.exists(REF_LIB):  # the reference's own CUDA kernels under the same host: how far THEY sit from the oracle
    CFG1_VARIANTS.append(("refkernels", dict(fused=False, kernel_lib=REF_LIB), 16))


@pytest.mark.parametrize("name,kw,steps", CFG1_VARIANTS)
def test_qwen3_4b_config1_vs_live_oracle(w4b, cfg1_oracle, name, kw, steps):
    if cfg1_oracle is None:  # host too slow for the live run: the committed fixture of the same configuration
        fx = F.Fixture(F.fixture_path("qwen3-4b", 128, 1))
        assert F.torch_weights_crc(w4b) == fx.meta["weights_crc"]
        m = _model(w4b, num_pages=64, **kw)
        got = _teacher_forced(m, synthetic_prompt(128), fx.tokens)
        m.close()
        for step, g in enumerate(got):
            ok, info = fx.compare(step, g, TOL_ULP)
            assert ok, f"{name} config-1 (fixture) step {step}: {info}"
        return
    want, toks = cfg1_oracle
    n = len(toks) if steps is None else min(steps, len(toks))
    m = _model(w4b, num_pages=64, **kw)
    got = _teacher_forced(m, synthetic_prompt(128), toks[:n])
    worst, same, same_at = 0.0, 0, []
    for step, (g, w_) in enumerate(zip(got, want[:n + 1])):
        ok, info = logits_agree(g, w_, TOL_ULP)
        worst = max(worst, info["err"] / (info["tol"] / TOL_ULP))
        same += info["same_argmax"]
        same_at.append(bool(info["same_argmax"]))
        assert ok, f"{name} config-1 step {step}: {info}"
    # free-running greedy sequence vs the oracle's: reported, and must at least start together
    free, _, _ = m.generate(synthetic_prompt(128), n + 1)
    m.close()
    oracle_seq = toks[:n] + [O.argmax(want[n])]
    div = next((i for i, (a, b) in enumerate(zip(free, oracle_seq)) if a != b), None)
    print(f"\n[fullsize] {name} config 1: {n + 1} steps, worst |dlogit| = {worst:.2f} ulp(rowmax), arg-max equal "
          f"{same}/{n + 1}, free-running first divergence: {div}")
    # Up to the first divergence the free-running and the teacher-forced runs see the same tokens, so a divergence at
    # step `div` must be one of the near-ties the parity rule accepted there (top-1/top-2 gap <= 2 tol); anything else
    # would mean generate() and the step-by-step path disagree.
    assert div is None or not same_at[div], (div, same_at)


@pytest.mark.parametrize("name,kw", [("fused", dict(fused=True)), ("compat", dict(fused=False))])
def test_qwen3_4b_config2_vs_fixture(w4b, name, kw):
    path = F.fixture_path("qwen3-4b", 2048, 1)
    assert os.path.exists(path), f"{path} missing: run tests/golden/make_parity_fixtures.py"
    fx = F.Fixture(path)
    assert F.torch_weights_crc(w4b) == fx.meta["weights_crc"], \
        "the CPU generator produced a different checkpoint than the fixture's: regenerate the fixture"
    m = _model(w4b, num_pages=2200 // 16 + 8, **kw)
    got = _teacher_forced(m, synthetic_prompt(2048), fx.tokens)
    m.close()
    worst, same = 0.0, 0
    for step, g in enumerate(got):
        ok, info = fx.compare(step, g, TOL_ULP)
        worst = max(worst, info["err_ulp_rowmax"])
        same += info["same_argmax"]
        assert ok, f"{name} config-2 step {step}: {info}"
    print(f"\n[fullsize] {name} config 2 (2048-token prefill + {len(fx.tokens)} decode steps): worst |dlogit| = "
          f"{worst:.2f} ulp(rowmax), arg-max equal {same}/{len(got)}")
