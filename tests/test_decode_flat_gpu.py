"""Decode attention of many requests (csrc/decode_attention_flat.cu): runs of pages that begin and end inside requests, on their borders, with several
requests to a run and one request over many, more requests than a warp has lanes, requests without a page, V before K in the pool, and places and counters
used again."""
import ctypes as C  # noqa: F401
import math

import pytest
import torch

from pegainfer_b200 import ffi

pytestmark = pytest.mark.gpu
NQ, NKV, HD, PS = 32, 8, 128, 16


@pytest.fixture(scope="module")
def lib():
    l = ffi.lib()
    l.cuda_set_device(0)
    l.cublas_init()
    return l


def rope(x, cos, sin):
    a, b = x.chunk(2, -1)
    return (x.float() * cos[:, None].float() + torch.cat([-b, a], -1).float() * sin[:, None].float()).bfloat16()


def normed(x, w):  # the rounding points of qk_norm_rope.cu
    inv = torch.rsqrt(x.float().square().mean(-1, keepdim=True) + 1e-6)
    return ((x.float() * inv).bfloat16().float() * w.float()).bfloat16()


def check(lib, lens, v_first=False, empty=(), rounds=1, places=37):
    """empty: requests without a page (their length is taken for zero)"""
    g = torch.Generator(device="cuda").manual_seed(sum(lens) + len(lens))
    rn = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731
    lens = [0 if i in empty else n for i, n in enumerate(lens)]
    bs, need = len(lens), [(n + PS - 1) // PS for n in lens]
    order = (torch.randperm(sum(need), generator=g, device="cuda") + 1).tolist()
    ptr = [0]
    for m in need:
        ptr.append(ptr[-1] + m)
    pool = torch.full((sum(need) + 2, 2, PS, NKV, HD), float("nan"), device="cuda").bfloat16()
    kx, vx = (1, 0) if v_first else (0, 1)
    ctx = []
    for i, n in enumerate(lens):
        full = torch.full((2, need[i] * PS, NKV, HD), float("nan"), device="cuda").bfloat16()
        if n:
            full[:, :n - 1] = rn(2, n - 1, NKV, HD).bfloat16()
        ctx.append(full)
        for j in range(need[i]):
            pool[order[ptr[i] + j], kx], pool[order[ptr[i] + j], vx] = full[0, j * PS:(j + 1) * PS], full[1, j * PS:(j + 1) * PS]
    q, k, v = rn(bs, NQ, HD).bfloat16(), rn(bs, NKV, HD).bfloat16(), rn(bs, NKV, HD).bfloat16()
    qw, kw = (1 + 0.1 * rn(HD)).bfloat16(), (1 + 0.1 * rn(HD)).bfloat16()
    inv = 1e6 ** (-torch.arange(0, HD, 2, device="cuda") / HD)
    ang = torch.arange(4096, device="cuda")[:, None] * inv
    cos, sin = torch.cat([ang.cos()] * 2, 1).bfloat16(), torch.cat([ang.sin()] * 2, 1).bfloat16()
    pos = i32([max(n - 1, 0) for n in lens])
    last, order_d, ptr_d = i32([(n - 1) % PS + 1 if n else 0 for n in lens]), i32(order), i32(ptr)
    partial, counters = torch.full((bs * places * NQ * (HD + 2),), float("nan"), device="cuda"), torch.zeros(bs * NKV, dtype=torch.int32, device="cuda")
    half, before = PS * NKV * HD, pool.clone()
    got = []
    for _ in range(rounds):
        out = torch.full((bs + 1, NQ, HD), 7.0, device="cuda").bfloat16()
        assert lib.pk_b200_decode_attention_fused(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), pool.data_ptr(), half * kx, half * vx,
                                                  order_d.data_ptr(), ptr_d.data_ptr(), last.data_ptr(), pos.data_ptr(), qw.data_ptr(), kw.data_ptr(),
                                                  cos.data_ptr(), sin.data_ptr(), 1e-6, partial.data_ptr(), counters.data_ptr(), 64, places, NQ, NKV, HD, PS,
                                                  bs, 2 * half, HD ** -0.5, None) == 0
        torch.cuda.synchronize()
        assert (out[bs] == 7.0).all() and lib.pk_b200_wait_errors() == 0 and not counters.any()
        got.append(out[:bs].clone())
    assert all(torch.equal(x, got[0]) for x in got)
    at = pos.long()
    qr, kr = rope(normed(q, qw), cos[at], sin[at]), rope(normed(k, kw), cos[at], sin[at])
    for i, n in enumerate(lens):
        if not n:
            assert not got[0][i].any()
            continue
        page, row = order[ptr[i] + (n - 1) // PS], (n - 1) % PS
        new_k = pool[page, kx, row].float()
        # one bf16 rounding of the norm and one of the rotation may fall to the other side
        assert ((new_k - kr[i].float()).abs() <= 2 ** -6 * kr[i].float().abs() + 2 ** -7).all() and torch.equal(pool[page, vx, row], v[i])
        before[page, :, row] = pool[page, :, row]
        keys, vals = ctx[i][0, :n].double(), ctx[i][1, :n].double()
        keys[n - 1], vals[n - 1] = new_k.double(), v[i].double()
        for h in range(NQ):
            p = torch.softmax(keys[:, h // 4] @ qr[i, h].double() * HD ** -0.5, 0)
            want = p @ vals[:, h // 4]
            # q as the kernel rounds it may be an ulp off in single entries (scores move by 2^-8 of their spread); the result is rounded once
            assert (got[0][i, h].double() - want).norm() <= 2 ** -6 * want.norm() + 1e-3, (i, h)
    assert torch.equal(pool.nan_to_num(), before.nan_to_num())  # nothing else was written


@pytest.mark.parametrize("lens", [
    [16] * 19, [1] * 24, [17] * 37, [4000] + [1] * 20, [1] * 20 + [4000], [300 + 7 * i for i in range(25)], [16 * (i + 1) for i in range(24)],
    [33] * 70, [2048] * 19, [5, 900, 16, 2047, 31, 32, 64] * 5])
def test_against_64_bits(lib, lens):
    check(lib, lens, rounds=2)


def test_values_before_keys(lib):
    check(lib, [100 + 31 * i for i in range(20)], v_first=True)


@pytest.mark.parametrize("empty", [(0,), (19,), (3, 4, 5, 12), tuple(range(0, 40, 2)), tuple(range(33))])
def test_requests_without_a_page(lib, empty):
    check(lib, [60 + 17 * i for i in range(40)], empty=empty)


def test_too_few_places_go_to_the_other_kernel(lib):
    check(lib, [40 * i + 1 for i in range(20)], places=1)
