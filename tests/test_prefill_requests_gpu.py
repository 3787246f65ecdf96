"""Prompt attention of many requests, whose CTAs look for their pair of query tiles a request per lane: fewer requests than lanes, as many, more, requests of one
tile and of several, behind cached keys.  The rows of a request are the bits of a call with that request alone, and near those in 64 bits."""
import math

import pytest
import torch

from pegainfer_b200 import ffi

pytestmark = pytest.mark.gpu
F64 = torch.float64
HD, PAGE = 128, 16


@pytest.fixture(scope="module")
def lib():
    l = ffi.lib()
    l.cuda_set_device(0)
    l.cublas_init()
    return l


@pytest.mark.parametrize("starts,lens,nq,nkv", [
    ([0], [300], 32, 8), ([0, 0, 0], [411, 256, 198], 32, 8), ([0, 9] * 16, [257, 3] * 16, 8, 2), ([5] * 33, [40] * 33, 8, 2), ([0] * 40, [1 + 37 * i for i in range(40)], 8, 2), ([0, 300] * 30, [128, 140] * 30, 32, 8),
    ([2000, 0] * 20, [1, 256] * 20, 16, 4), ([100] * 70, [129] * 70, 4, 4)])
def test_alone_and_against_64_bits(lib, starts, lens, nq, nkv):
    n, T = len(lens), sum(lens)
    g = torch.Generator(device="cuda").manual_seed(T)
    need = [(s + m + PAGE - 1) // PAGE for s, m in zip(starts, lens)]
    order = torch.randperm(sum(need), generator=g, device="cuda").to(torch.int32)
    kv = torch.randn(sum(need), 2, PAGE, nkv, HD, generator=g, device="cuda").bfloat16()  # a page: keys, values
    q = (1.5 * torch.randn(T, nq, HD, generator=g, device="cuda")).bfloat16()
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731
    first, row0 = [sum(need[:i]) for i in range(n + 1)], [sum(lens[:i]) for i in range(n + 1)]
    last = [(s + m - 1) % PAGE + 1 for s, m in zip(starts, lens)]

    def run(a, b):  # requests a .. b - 1
        rows = q[row0[a]:row0[b]].contiguous()
        out = torch.full((len(rows) + 1, nq, HD), 9.0, device="cuda").bfloat16()
        pages, indptr, lpl, qptr = order[first[a]:first[b]].contiguous(), i32([x - first[a] for x in first[a:b + 1]]), i32(last[a:b]), i32([x - row0[a] for x in row0[a:b + 1]])
        assert lib.pk_b200_prefill_attention_tc(rows.data_ptr(), out.data_ptr(), kv.data_ptr(), 0, PAGE * nkv * HD, pages.data_ptr(), indptr.data_ptr(), lpl.data_ptr(),
                                                qptr.data_ptr(), nq, nkv, HD, PAGE, len(rows), b - a, 2 * PAGE * nkv * HD, HD ** -0.5, None) == 0
        torch.cuda.synchronize()
        assert (out[-1] == 9.0).all() and lib.pk_b200_wait_errors() == 0
        return out[:-1]

    got = run(0, n)
    for i, (s, m) in enumerate(zip(starts, lens)):
        rows = got[row0[i]:row0[i + 1]]
        if n > 1:
            assert torch.equal(rows, run(i, i + 1)), i
        keys = kv[order[first[i]:first[i + 1]].long()].transpose(0, 1).reshape(2, -1, nkv, HD)[:, :s + m].to(F64)
        hidden = torch.arange(s + m, device="cuda")[None] > torch.arange(s, s + m, device="cuda")[:, None]
        for h in range(0, nq, 3):
            sc = q[row0[i]:row0[i + 1], h].to(F64) @ keys[0, :, h * nkv // nq].T / math.sqrt(HD)
            p = torch.softmax(sc.masked_fill(hidden, -math.inf), -1)
            want, size = p @ keys[1, :, h * nkv // nq], p @ keys[1, :, h * nkv // nq].abs()
            # weights and result are rounded to bf16 once each, the denominator is that of the rounded weights
            assert ((rows[:, h].to(F64) - want).abs() <= 2 ** -8 * size + 2 ** -8 * want.abs() + 1e-4).all(), (i, h)
