"""Grouped-query attention of 64 rows and more whose (tile, head) pairs leave SMs idle (clusters that share the keys), against the per-head softmax in 64 bits:
cluster sizes 2, 4 and 8, tiles that end inside a request and hold several, a last tile of few rows, shares without a key, windows, kept first keys, chunks,
soft cap, distance bias, gates per entry and per head, rows with and without a sink; and next to it the same rows where no cluster is used."""
import ctypes as C
import math

import pytest
import torch

from pegainfer_b200 import ffi

pytestmark = pytest.mark.gpu
BF16, F64 = torch.bfloat16, torch.float64
PAGE = 16


@pytest.fixture(scope="module")
def lib():
    l = ffi.lib()
    l.cuda_set_device(0)
    l.cublas_init()
    return l


@pytest.mark.parametrize("lens,had,H,G,D,opt", [
    ([64], [0], 1, 1, 32, {}), ([64], [1000], 2, 1, 128, {}), ([100, 1, 30], [700, 0, 2000], 4, 2, 64, {"sink": 1}), ([65], [3000], 2, 2, 96, {"gate": 1}),
    ([40, 40, 40], [600, 900, 30], 4, 1, 128, {"window": 300}), ([130], [1500], 8, 2, 64, {"window": 200, "keep": 70, "gate": 2}),
    ([200], [800], 4, 4, 64, {"chunk": 256, "sink": 1}), ([90], [1200], 6, 3, 128, {"softcap": 20.0, "slope": 8.0}), ([700], [0], 2, 1, 64, {}), ([1300, 5], [0, 4], 16, 4, 64, {})])
def test_against_64_bits(lib, lens, had, H, G, D, opt):
    T, n = sum(lens), len(lens)
    g = torch.Generator(device="cuda").manual_seed(T + H + D)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda").to(BF16)  # noqa: E731
    need = [(a + b + PAGE - 1) // PAGE for a, b in zip(lens, had)]
    order = torch.randperm(sum(need), generator=g, device="cuda").to(torch.int32)
    off = [sum(need[:i]) for i in range(n)]
    cache, q = r(sum(need), PAGE, 2 * G * D), r(T, H * D)
    pos = torch.tensor([b + i for a, b in zip(lens, had) for i in range(a)], dtype=torch.int32, device="cuda")
    req = torch.tensor([i for i, a in enumerate(lens) for _ in range(a)], dtype=torch.int32, device="cuda")
    offs = torch.tensor(off, dtype=torch.int32, device="cuda")
    sink = r(H) if opt.get("sink") else None
    gate = r(T, H if opt.get("gate") == 2 else H * D) if opt.get("gate") else None
    w, keep, chunk, cap, slope = (opt.get(k, 0) for k in ("window", "keep", "chunk", "softcap", "slope"))
    out = torch.full((T, H * D), float("nan"), dtype=BF16, device="cuda")
    x = ffi.AttnExtra(window=w, softcap=float(cap), slope_log2=float(slope), gate=gate.data_ptr() if gate is not None else None, gate_ld=gate.shape[1] if gate is not None else 0,
                      max_kv_len=max(a + b for a, b in zip(lens, had)), keep_first=keep, gate_per_head=int(opt.get("gate") == 2))
    assert lib.pk_gqa_attention_ex(q.data_ptr(), cache.data_ptr(), sink.data_ptr() if sink is not None else None, pos.data_ptr(), req.data_ptr(), offs.data_ptr(),
                                   order.data_ptr(), out.data_ptr(), PAGE * 2 * G * D, PAGE, T, H, G, D, D, D ** -0.5, chunk, C.byref(x), 0, None) == 0
    torch.cuda.synchronize()
    row = 0
    for i, (a, b) in enumerate(zip(lens, had)):
        kv = cache[order[off[i]:off[i] + need[i]].long()].reshape(-1, 2, G, D)[:a + b].to(F64)
        at, j = torch.arange(b, b + a, device="cuda")[:, None], torch.arange(a + b, device="cuda")[None]
        lo = torch.zeros_like(at)
        if chunk:
            lo = at // chunk * chunk
        if w:
            lo = torch.maximum(lo, at - w + 1)
        hidden = (j > at) | ((j < lo) & ~((j < keep) if w else torch.zeros_like(j, dtype=torch.bool)))
        for h in range(H):
            s = q[row:row + a].view(a, H, D)[:, h].to(F64) @ kv[:, 0, h * G // H].T * D ** -0.5
            if cap:
                s = cap * torch.tanh(s / cap)
            if slope:
                s = s - 2.0 ** (-slope * (h + 1) / H) * (at - j)
            s = s.masked_fill(hidden, -math.inf)
            if sink is not None:
                s = torch.cat([s, sink[h].to(F64).expand(a, 1)], 1)
            p = torch.softmax(s, -1)[:, :a + b]
            o = p @ kv[:, 1, h * G // H]
            if gate is not None:
                o = o * torch.sigmoid(gate[row:row + a].to(F64)[:, h:h + 1] if opt["gate"] == 2 else gate[row:row + a].view(a, H, D)[:, h].to(F64))
            got = out[row:row + a].view(a, H, D)[:, h].to(F64)
            # P rounded to bf16 against a running maximum (2^-8 of each weight, of either sign) and one rounding of the result
            assert (got - o).norm() <= 6e-3 * o.norm() and (got - o).abs().max() <= 2 ** -7 * kv[:, 1].abs().max(), (i, h)
        row += a
