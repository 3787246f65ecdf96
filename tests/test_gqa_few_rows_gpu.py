"""Grouped-query attention of fewer than 64 rows (gqa_decode_kernel in csrc/gqa_attention.cu): groups that fill a tile of 16 rows and groups that do not,
portions around the tokens of a tile, decoded tokens and portions in one step, contexts around the 16-key tiles and the warps' turns, clusters of one to eight
CTAs, and every option of the scores, against 64 bits; unused slots of the cache hold NaN."""
import ctypes as C

import pytest
import torch

from pegainfer_b200 import ffi

pytestmark = pytest.mark.gpu
PS = 16


@pytest.fixture(scope="module")
def lib():
    l = ffi.lib()
    l.cuda_set_device(0)
    l.cublas_init()
    return l


def check(lib, steps, H, G, D, window=0, chunk=0, softcap=0.0, keep=0, slope=0.0, sink=True, gate=None, known=True):
    """steps: (tokens, already cached) of every request"""
    g = torch.Generator(device="cuda").manual_seed(H * 1000 + D + sum(a * 7 + b for a, b in steps))
    rn = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731
    need = [(a + b + PS - 1) // PS for a, b in steps]
    order = torch.randperm(sum(need), generator=g, device="cuda").tolist()
    cache = torch.full((sum(need) + 1, PS, 2 * G * D), float("nan"), device="cuda").bfloat16()
    off, at, ctx = [], 0, []
    for (a, b), m in zip(steps, need):
        rows = rn(a + b, 2 * G * D).bfloat16()
        full = torch.full((m * PS, 2 * G * D), float("nan"), device="cuda").bfloat16()
        full[:a + b] = rows
        for j in range(m):
            cache[order[at + j]] = full[j * PS:(j + 1) * PS]
        off.append(at)
        at += m
        ctx.append(rows.double())
    T = sum(a for a, _ in steps)
    q, sk = (1.5 * rn(T, H, D)).bfloat16(), rn(H).bfloat16()
    gt = rn(T, H if gate == "head" else H * D).bfloat16()
    pos, req = i32([b + j for a, b in steps for j in range(a)]), i32([r for r, (a, _) in enumerate(steps) for _ in range(a)])
    off_d, pages = i32(off), i32(order)
    out = torch.full((T + 1, H, D), 5.0, device="cuda").bfloat16()
    ex = ffi.AttnExtra(window=window, softcap=softcap, slope_log2=slope, keep_first=keep, gate=gt.data_ptr() if gate else None, gate_ld=gt.shape[1],
                       gate_per_head=int(gate == "head"), max_kv_len=max(a + b for a, b in steps) if known else 0)
    scale = D ** -0.5
    assert lib.pk_gqa_attention_ex(q.data_ptr(), cache.data_ptr(), sk.data_ptr() if sink else None, pos.data_ptr(), req.data_ptr(), off_d.data_ptr(),
                                   pages.data_ptr(), out.data_ptr(), PS * 2 * G * D, PS, T, H, G, D, D, scale, chunk, C.byref(ex), 0, None) == 0
    torch.cuda.synchronize()
    assert (out[T] == 5.0).all()
    row = 0
    for (a, b), rows in zip(steps, ctx):
        p, j = torch.arange(b, b + a, device="cuda")[:, None], torch.arange(a + b, device="cuda")[None]
        lo = (p // chunk * chunk) if chunk else torch.zeros_like(p)
        if window:
            lo = torch.maximum(lo, p - window + 1)
        seen = (j <= p) & ((j >= lo) | (j < (keep if window else 0)))
        for h in range(H):
            k, v = rows[:, h * G // H * D:(h * G // H + 1) * D], rows[:, (G + h * G // H) * D:(G + h * G // H + 1) * D]
            s = q[row:row + a, h].double() @ k.T * scale
            if softcap:
                s = softcap * torch.tanh(s / softcap)
            if slope:
                s = s - 2.0 ** (-slope * (h + 1) / H) * (p - j)
            s = s.masked_fill(~seen, -float("inf"))
            if sink:
                s = torch.cat([s, sk[h].double().expand(a, 1)], 1)
            w = torch.softmax(s, -1)[:, :a + b]
            f = torch.ones((), dtype=torch.float64, device="cuda")
            if gate:
                f = torch.sigmoid(gt[row:row + a, h:h + 1].double() if gate == "head" else gt[row:row + a, h * D:(h + 1) * D].double())
            want, got = w @ v * f, out[row:row + a, h].double()
            # weights and the result are rounded to bf16 once each; fast exponentials and the cap's reciprocal stay below 1e-5 of the largest weight
            bound = (2 ** -8 + 1e-4) * (w @ v.abs()) * f + 2 ** -8 * want.abs() + 1e-4
            assert ((got - want).abs() <= bound).all(), (a, b, h, (got - want).abs().max().item())
        row += a


@pytest.mark.parametrize("H,G,D", [(16, 4, 128), (8, 8, 64), (16, 8, 96), (6, 2, 32), (10, 2, 64), (24, 3, 128), (16, 1, 128)])
@pytest.mark.parametrize("steps", [
    [(1, 0)], [(1, 15)], [(1, 16), (1, 63), (1, 64), (1, 200)], [(1, 2500)], [(3, 0), (5, 17), (4, 300)], [(17, 30), (1, 511), (1, 0), (16, 1)],
    [(63, 0)], [(40, 700), (23, 5)], [(1, 9 * i) for i in range(63)], [(1, 1000), (4, 900), (1, 1000)]])
def test_steps(lib, H, G, D, steps):
    check(lib, steps, H, G, D)


@pytest.mark.parametrize("opts", [
    dict(window=100), dict(window=1, sink=False), dict(chunk=64), dict(window=70, keep=5), dict(window=33, keep=40, softcap=20.0), dict(softcap=30.0, sink=False),
    dict(slope=8.0), dict(gate="entry"), dict(gate="head", window=150), dict(known=False), dict(window=300, chunk=128, slope=4.0, gate="entry", softcap=50.0)])
@pytest.mark.parametrize("steps", [[(1, 400), (1, 31), (1, 129)], [(6, 130), (1, 64), (9, 0), (20, 250)]])
def test_options(lib, steps, opts):
    check(lib, steps, 8, 2, 64, **opts)
    check(lib, steps, 16, 4, 128, **opts)


@pytest.mark.parametrize("H,G,D", [(16, 4, 128), (8, 8, 64), (16, 8, 96), (6, 2, 32), (24, 3, 128), (16, 1, 128)])
@pytest.mark.parametrize("steps", [[(24, 2500)], [(8, 4200)], [(1, 6000)], [(60, 900)], [(9, 2600), (1, 9), (3, 0)], [(20, 130), (1, 3000), (30, 97), (12, 800)]])
def test_requests_that_run_in_tiles(lib, H, G, D, steps):
    """several tokens behind many keys: a request's clusters become the CTAs of tiles of 64 rows, beside requests that run by themselves"""
    check(lib, steps, H, G, D)
    check(lib, steps, H, G, D, window=700, keep=9, softcap=25.0, gate="entry")
    check(lib, steps, H, G, D, chunk=512, slope=6.0, sink=False, gate="head", known=False)


def test_more_heads_to_a_group_than_a_tile_has_rows(lib):
    check(lib, [(1, 300), (7, 20)], 40, 2, 64)
