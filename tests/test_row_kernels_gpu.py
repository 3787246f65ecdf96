"""Norms of rows, the rotation of heads and the gated norm of heads at the edges of their launch shapes: the last lane's pieces, odd numbers of rows and heads, the
switch between eight and four warps a row, rows just too long; against 64 bits."""
import pytest
import torch

from pegainfer_b200 import ffi

pytestmark = pytest.mark.gpu
BF16, F64 = torch.bfloat16, torch.float64
EPS = 1e-6


@pytest.fixture(scope="module")
def lib():
    l = ffi.lib()
    l.cuda_set_device(0)
    l.cublas_init()
    return l


def rnd(g, *s):
    return torch.randn(*s, generator=g, device="cuda").to(BF16)


def near(got, want):  # one rounding to bf16 of a value that fp32 holds to 1e-6
    return ((got.to(F64) - want).abs() <= want.abs() * (2 ** -8 + 1e-5) + 1e-30).all()


@pytest.mark.parametrize("dim", [8, 264, 1024, 2048, 2056, 3072, 3080, 4096, 4104])
@pytest.mark.parametrize("rows", [1, 3, 295, 297])
def test_norms(lib, dim, rows):
    g = torch.Generator(device="cuda").manual_seed(dim + rows)
    x, r, w = rnd(g, rows, dim), rnd(g, rows, dim), rnd(g, dim)
    n = lambda v: v * torch.rsqrt(v.square().mean(-1, keepdim=True) + EPS)  # noqa: E731
    out, one, hidden, added = (torch.full_like(x, float("nan")) for _ in range(4))
    hidden.copy_(x)
    lib.rms_norm_batched_cuda(x.data_ptr(), w.data_ptr(), out.data_ptr(), dim, rows, EPS, None)
    lib.rms_norm_batched_offset_cuda(x.data_ptr(), w.data_ptr(), one.data_ptr(), dim, rows, EPS, None)
    lib.fused_add_rms_norm_batched_cuda(hidden.data_ptr(), r.data_ptr(), w.data_ptr(), added.data_ptr(), dim, rows, EPS, None)
    torch.cuda.synchronize()
    h = x.to(F64) + r.to(F64)
    assert near(out, n(x.to(F64)) * w.to(F64)) and near(one, n(x.to(F64)) * (1 + w.to(F64)))
    assert torch.equal(hidden, h.to(BF16)) and near(added, n(h) * w.to(F64))


@pytest.mark.parametrize("nq,nkv,tokens", [(1, 0, 1), (0, 3, 5), (5, 2, 7), (32, 8, 600), (7, 2, 2300)])
def test_qk_norm_and_rotation(lib, nq, nkv, tokens):
    g = torch.Generator(device="cuda").manual_seed(nq + tokens)
    q, k, qw, kw = rnd(g, tokens, nq, 128), rnd(g, tokens, nkv, 128), rnd(g, 128), rnd(g, 128)
    ang = torch.arange(4096, device="cuda")[:, None] * 1e4 ** (-torch.arange(64, device="cuda") / 64)
    cos, sin = torch.cat([ang.cos()] * 2, 1).to(BF16), torch.cat([ang.sin()] * 2, 1).to(BF16)
    pos = torch.randint(0, 4096, (tokens,), generator=g, device="cuda", dtype=torch.int32)
    want = []
    for x, w in ((q, qw), (k, kw)):
        f = x.float()
        t = (f * torch.rsqrt(f.square().mean(-1, keepdim=True) + EPS)).to(BF16)
        t = (t.float() * w.float()).to(BF16).to(F64)  # the two roundings in between
        lo, hi, c, s = t[..., :64], t[..., 64:], cos[pos.long(), None, :64].to(F64), sin[pos.long(), None, :64].to(F64)
        want.append(torch.cat([lo * c - hi * s, lo * s + hi * c], -1))
    lib.qk_norm_rope_batched_decode_cuda(q.data_ptr(), k.data_ptr(), qw.data_ptr(), kw.data_ptr(), cos.data_ptr(), sin.data_ptr(), pos.data_ptr(), nq, nkv, 128,
                                         tokens, EPS, None)
    torch.cuda.synchronize()
    for got, w in zip((q, k), want):
        # an intermediate rounding that falls the other way moves a partner by 2^-8 of itself
        assert w.numel() == 0 or ((got.to(F64) - w).abs() <= w.abs() * 2 ** -8 + w.abs().amax(-1, keepdim=True) * 2 ** -7).all()
        assert w.numel() == 0 or (got.to(F64) - w).norm() <= 3e-3 * w.norm()


@pytest.mark.parametrize("heads", [1, 15, 33, 9471, 9473])
def test_gated_norm_of_heads(lib, heads):
    g = torch.Generator(device="cuda").manual_seed(heads)
    x, gate, w = rnd(g, heads, 128), 8 * rnd(g, heads, 128), torch.randn(128, generator=g, device="cuda")
    gate[0, :4] = torch.tensor([120.0, -120.0, 0.0, -60.0])
    out = torch.zeros_like(x)
    lib.rms_norm_gated_cuda(x.data_ptr(), w.data_ptr(), gate.data_ptr(), out.data_ptr(), heads, 128, EPS, None)
    torch.cuda.synchronize()
    v, z = x.to(F64), gate.to(F64)
    assert near(out, v * torch.rsqrt(v.square().mean(-1, keepdim=True) + EPS) * w.to(F64) * z * torch.sigmoid(z))
