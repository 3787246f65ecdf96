"""Row kernels add squares in a stated order, so that a row has the same bits from whichever form of a kernel takes it: compared bit for bit with the same fp32
operations in torch (squares of bf16 are exact in fp32, so a chain of fused multiply-adds is a chain of additions)."""
import pytest
import torch

from pegainfer_b200 import ffi

pytestmark = pytest.mark.gpu
BF16, F32 = torch.bfloat16, torch.float32
EPS = 1e-6


@pytest.fixture(scope="module")
def lib():
    l = ffi.lib()
    l.cuda_set_device(0)
    l.cublas_init()
    return l


def rnd(g, *s):
    return torch.randn(*s, generator=g, device="cuda").to(BF16)


def halves(s):
    """sum over the last axis (a power of two) by exchanges at half the distance each time"""
    while s.shape[-1] > 1:
        n = s.shape[-1] // 2
        s = s[..., :n] + s[..., n:]
    return s[..., 0]


def chain(sq):
    """the last axis one after the other"""
    s = torch.zeros_like(sq[..., 0])
    for i in range(sq.shape[-1]):
        s = s + sq[..., i]
    return s


@pytest.mark.parametrize("nq,nkv,tokens", [(3, 1, 2500), (16, 3, 900), (32, 8, 3333)])
def test_qk_norm_and_rotation(lib, nq, nkv, tokens):
    g = torch.Generator(device="cuda").manual_seed(nq + tokens)
    q, k, qw, kw = rnd(g, tokens, nq, 128), rnd(g, tokens, nkv, 128), rnd(g, 128), rnd(g, 128)
    ang = torch.arange(4096, device="cuda")[:, None] * 1e4 ** (-torch.arange(64, device="cuda") / 64)
    cos, sin = torch.cat([ang.cos()] * 2, 1).to(BF16), torch.cat([ang.sin()] * 2, 1).to(BF16)
    pos = torch.randint(0, 4096, (tokens,), generator=g, device="cuda", dtype=torch.int32)
    c, s = (t[pos.long(), None, :64].to(F32) for t in (cos, sin))
    want = []
    for x, w in ((q, qw), (k, kw)):
        v = x.to(F32)
        r = torch.rsqrt(halves(chain(v.square().unflatten(-1, (16, 8)))) / 128 + EPS)  # sixteen chains of eight
        t = ((v * r[..., None]).to(BF16).to(F32) * w.to(F32)).to(BF16).to(F32)
        lo, hi = t[..., :64], t[..., 64:]
        want.append(torch.cat([lo * c - hi * s, lo * s + hi * c], -1).to(BF16))
    lib.qk_norm_rope_batched_decode_cuda(q.data_ptr(), k.data_ptr(), qw.data_ptr(), kw.data_ptr(), cos.data_ptr(), sin.data_ptr(), pos.data_ptr(), nq, nkv, 128,
                                         tokens, EPS, None)
    torch.cuda.synchronize()
    assert torch.equal(q, want[0]) and torch.equal(k, want[1])


@pytest.mark.parametrize("offset", [4, 8])
def test_qk_norm_on_eight_byte_boundaries(lib, offset):
    """pointers on 8-byte boundaries take the same pieces in two halves"""
    g = torch.Generator(device="cuda").manual_seed(offset)
    nq, nkv, tokens = 5, 2, 70
    q, k, qw, kw = rnd(g, tokens, nq, 128), rnd(g, tokens, nkv, 128), rnd(g, 128), rnd(g, 128)
    cos, sin = rnd(g, 256, 128), rnd(g, 256, 128)
    pos = torch.randint(0, 256, (tokens,), generator=g, device="cuda", dtype=torch.int32)

    def moved(t):
        room = torch.empty(t.numel() + offset, dtype=BF16, device="cuda")[offset:]
        return room.copy_(t.flatten()).view(t.shape)
    a, b = [t.clone() for t in (q, k)], [moved(t) for t in (q, k)]
    for (x, y), t in ((a, (qw, kw, cos, sin)), (b, [moved(t) for t in (qw, kw, cos, sin)])):
        lib.qk_norm_rope_batched_decode_cuda(x.data_ptr(), y.data_ptr(), t[0].data_ptr(), t[1].data_ptr(), t[2].data_ptr(), t[3].data_ptr(), pos.data_ptr(), nq,
                                             nkv, 128, tokens, EPS, None)
    torch.cuda.synchronize()
    assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])


def norm_sum(sq, few):
    """of rows [n, dim] of squares.  A row by itself: chains of eight elements, by exchange within 32 of them, then so between the warps; many rows: lane l
    takes its pieces l, l + 32, .. one after the other, then by exchange"""
    pieces = sq.unflatten(-1, (-1, 8))
    if few:
        s = torch.nn.functional.pad(chain(pieces), (0, 1024 - pieces.shape[-2])).unflatten(-1, (32, 32))
        return halves(halves(s))
    pieces = torch.nn.functional.pad(pieces, (0, 0, 0, -pieces.shape[-2] % 32)).unflatten(-2, (-1, 32))
    return halves(chain(pieces.transpose(-3, -2).flatten(-2)))


@pytest.mark.parametrize("dim", [8, 1024, 1032, 2560, 2816, 4096])
@pytest.mark.parametrize("rows", [295, 297, 2051])
def test_norms(lib, dim, rows):
    sms, width = torch.cuda.get_device_properties(0).multi_processor_count, torch.full((1,), float(dim), device="cuda")  # (by a number: times its reciprocal)
    for seed in range(6 if rows < 300 else 1):  # (few sums fall where the order shows in bf16)
        g = torch.Generator(device="cuda").manual_seed(dim + rows + 7 * seed)
        x, r, w = rnd(g, rows, dim), rnd(g, rows, dim), rnd(g, dim)
        out, one, hidden, added = (torch.full_like(x, float("nan")) for _ in range(4))
        hidden.copy_(x)
        lib.rms_norm_batched_cuda(x.data_ptr(), w.data_ptr(), out.data_ptr(), dim, rows, EPS, None)
        lib.rms_norm_batched_offset_cuda(x.data_ptr(), w.data_ptr(), one.data_ptr(), dim, rows, EPS, None)
        lib.fused_add_rms_norm_batched_cuda(hidden.data_ptr(), r.data_ptr(), w.data_ptr(), added.data_ptr(), dim, rows, EPS, None)
        torch.cuda.synchronize()

        def scaled(v, weight):
            return (v * torch.rsqrt(norm_sum(v.square(), rows < 2 * sms) / width + EPS)[:, None] * weight).to(BF16)
        assert torch.equal(out, scaled(x.to(F32), w.to(F32)))
        assert torch.equal(one, scaled(x.to(F32), 1 + w.to(F32)))
        h = x.to(F32) + r.to(F32)
        assert torch.equal(hidden, h.to(BF16))
        # (the squares of these sums round: against a fused multiply-add a chain of additions is off by a last bit, which bf16 seldom shows)
        assert (added != scaled(h, w.to(F32))).float().mean() < 1e-4
