"""Decode attention of many requests (csrc/decode_attention_flat.cu): runs of pages that begin and end inside requests, on their borders, with several
requests to a run and one request over many, more requests than a warp has lanes, requests without a page, V before K in the pool, and places and counters
used again."""
import ctypes as C  # noqa: F401
import math

import pytest
import torch

from pegainfer_b200 import ffi

pytestmark = pytest.mark.gpu
NQ, NKV, HD, PS, MIN_PAGES = 32, 8, 128, 16, 2


@pytest.fixture(scope="module")
def lib():
    l = ffi.lib()
    l.cuda_set_device(0)
    l.cublas_init()
    return l


def check(lib, lens, v_first=False, empty=(), rounds=1, places=37, spare=()):
    """empty: requests without a page (their length is taken for zero); spare: requests whose last page holds no token yet (last_page_len 0)"""
    g = torch.Generator(device="cuda").manual_seed(sum(lens) + len(lens))
    rn = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731
    lens = [0 if i in empty else n for i, n in enumerate(lens)]
    lens = [(n + PS - 1) // PS * PS if i in spare else n for i, n in enumerate(lens)]
    bs, need = len(lens), [(n + PS - 1) // PS + (i in spare) for i, n in enumerate(lens)]
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
    last, order_d, ptr_d = i32([0 if i in spare else (n - 1) % PS + 1 if n else 0 for i, n in enumerate(lens)]), i32(order), i32(ptr)
    partial, counters = torch.full((bs * places * NQ * (HD + 2),), float("nan"), device="cuda"), torch.zeros(bs * NKV, dtype=torch.int32, device="cuda")
    # the kernel leaves states in `partial` where a request lies in several runs, as one of more pages than a run must; the cluster form never touches it
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    flat, run = bs * NKV > sms and bs * places >= 2 * sms, max((sum(need) + sms - 1) // sms, MIN_PAGES + 1)
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
        if max(need) > run or not flat:
            assert partial.isnan().all().item() != flat
        got.append(out[:bs].clone())
    assert all(torch.equal(x, got[0]) for x in got)
    qr, kr = q.clone(), k.clone()  # normed and rotated by the kernel of the same arithmetic (tested by itself)
    lib.qk_norm_rope_batched_decode_cuda(qr.data_ptr(), kr.data_ptr(), qw.data_ptr(), kw.data_ptr(), cos.data_ptr(), sin.data_ptr(), pos.data_ptr(), NQ, NKV, HD,
                                         bs, 1e-6, None)
    torch.cuda.synchronize()
    for i, n in enumerate(lens):
        if not n:
            assert not got[0][i].any()
            continue
        page, row = order[ptr[i] + (n - 1) // PS], (n - 1) % PS
        assert torch.equal(pool[page, kx, row], kr[i]) and torch.equal(pool[page, vx, row], v[i])
        before[page, :, row] = pool[page, :, row]
        keys, vals = ctx[i][0, :n].double(), ctx[i][1, :n].double()
        keys[n - 1], vals[n - 1] = kr[i].double(), v[i].double()
        for h in range(NQ):
            p = torch.softmax(keys[:, h // 4] @ qr[i, h].double() * HD ** -0.5, 0)
            want = p @ vals[:, h // 4]
            # The result is rounded to bf16 once (2^-8 of an entry).  Weights are held to 16 bits; an entry of q whose norm or rotation rounds the other way
            # than in the kernel that qr comes from (entries below 4: 2^-6, by a key's 2, by the scale 2^-3.5) moves them by 2^-8
            size, off = p @ vals[:, h // 4].abs(), (got[0][i, h].double() - want).abs()
            assert (off <= 2 ** -8 * (want.abs() + size)).all() and off.norm() <= 2 ** -8 * want.norm() + 2 ** -10 * size.norm(), (i, h)
    assert torch.equal(pool.nan_to_num(), before.nan_to_num())  # nothing else was written


@pytest.mark.parametrize("lens", [
    [16] * 19, [1] * 24, [17] * 37, [4000] + [1] * 20, [1] * 20 + [4000], [300 + 7 * i for i in range(25)], [16 * (i + 1) for i in range(24)],
    [33] * 70, [2048] * 19, [5, 900, 16, 2047, 31, 32, 64] * 5])
def test_against_64_bits(lib, lens):
    check(lib, lens, rounds=2)


def test_last_pages_without_a_token(lib):
    """a page that was taken ahead of its first token, first in a run, last in one and alone in one; what lies there (NaN) is not looked at"""
    check(lib, [100 + 31 * i for i in range(20)], spare=range(0, 20, 3))
    check(lib, [16] * 30, spare=range(30))


def test_values_before_keys(lib):
    check(lib, [100 + 31 * i for i in range(20)], v_first=True)


@pytest.mark.parametrize("empty", [(0,), (19,), (3, 4, 5, 12), tuple(range(0, 40, 2)), tuple(range(33))])
def test_requests_without_a_page(lib, empty):
    check(lib, [60 + 17 * i for i in range(40)], empty=empty)


def test_too_few_places_go_to_the_other_kernel(lib):
    check(lib, [40 * i + 1 for i in range(20)], places=1)
