"""Row kernels with wide loads (csrc/norm_rows.cuh, qk_norm_rope.cu, the conv and gated norm of qwen35_ops.cu) on both sides of their dispatch: row
counts around the change from a CTA to a warp per row, ragged row lengths, pointers off a 16-byte boundary, sequence lengths around a thread's tokens."""
import pytest
import torch

from pegainfer_b200 import ffi

pytestmark = pytest.mark.gpu
ULP = 2 ** -8  # one bf16 rounding, relative


@pytest.fixture(scope="module")
def lib():
    l = ffi.lib()
    l.cuda_set_device(0)
    return l


def rnd(seed, *shape, shift=0, scale=1.0):
    """bf16 tensor whose first element lies `shift` elements behind a 16-byte boundary"""
    g = torch.Generator(device="cuda").manual_seed(seed)
    n = 1
    for s in shape:
        n *= s
    buf = torch.zeros(n + 16, device="cuda", dtype=torch.bfloat16)
    buf[shift:shift + n] = torch.randn(n, generator=g, device="cuda") * scale
    return buf[shift:shift + n].view(*shape)


def near(got, want, ulps=1.0):
    # fp32 sums of up to 4104 squares and a reciprocal root add 2^-20 at most
    assert ((got.double() - want).abs() <= want.abs() * (ulps * ULP + 2 ** -20) + 1e-30).all()


@pytest.mark.parametrize("shift", [0, 4])
@pytest.mark.parametrize("dim", [8, 256, 1032, 2560, 2568, 4096, 4104])
@pytest.mark.parametrize("rows", [1, 295, 296, 301])
def test_norms(lib, rows, dim, shift):
    eps = 1e-6
    x, r, w = rnd(1, rows, dim, shift=shift), rnd(2, rows, dim, shift=shift), rnd(3, dim, scale=0.2)
    norm = lambda v, g: v * torch.rsqrt(v.square().mean(-1, keepdim=True) + eps) * g  # noqa: E731
    out = torch.zeros(rows + 1, dim, device="cuda").bfloat16()
    lib.rms_norm_batched_cuda(x.data_ptr(), w.data_ptr(), out.data_ptr(), dim, rows, eps, None)
    near(out[:rows], norm(x.double(), w.double()))
    lib.rms_norm_batched_offset_cuda(x.data_ptr(), w.data_ptr(), out.data_ptr(), dim, rows, eps, None)
    near(out[:rows], norm(x.double(), 1 + w.double()))
    s = x.double() + r.double()
    h = x.clone()
    lib.fused_add_rms_norm_batched_cuda(h.data_ptr(), r.data_ptr(), w.data_ptr(), out.data_ptr(), dim, rows, eps, None)
    near(out[:rows], norm(s.float().double(), w.double()))
    assert torch.equal(h, (x.float() + r.float()).bfloat16()) and (out[rows] == 0).all()


@pytest.mark.parametrize("shift", [0, 4])
@pytest.mark.parametrize("nq,nkv", [(32, 8), (5, 1), (1, 1)])
@pytest.mark.parametrize("tokens", [1, 7, 500])
def test_qk_norm_rope(lib, tokens, nq, nkv, shift):
    eps, start = 1e-6, 3
    q, k = rnd(4, tokens, nq, 128, shift=shift), rnd(5, tokens, nkv, 128, shift=shift)
    qw, kw = rnd(6, 128, shift=shift), rnd(7, 128, shift=shift)
    ang = torch.arange(tokens + start, device="cuda").float()[:, None] * (1e4 ** (-torch.arange(64, device="cuda") / 64.0))
    cos, sin = torch.cat([ang.cos()] * 2, 1).bfloat16(), torch.cat([ang.sin()] * 2, 1).bfloat16()

    def want(x, w):
        x = x.double()
        t = (x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps)).bfloat16().double() * w.double()
        t = t.bfloat16().double()
        c, s = cos[start:, None].double(), sin[start:, None].double()
        a, b = t.chunk(2, -1)
        return t * c + torch.cat([-b, a], -1) * s, t.abs()

    for x, w in ((q, qw), (k, kw)):
        x.want = want(x, w)
    lib.prefill_qk_norm_rope_only_cuda(q.data_ptr(), k.data_ptr(), qw.data_ptr(), kw.data_ptr(), cos.data_ptr(), sin.data_ptr(), nq, nkv, 128, tokens, start, eps,
                                       None)
    torch.cuda.synchronize()
    for x in (q, k):
        y, t = x.want
        # the two roundings before the rotation may fall the other way by an fp32 ulp of the norm: one bf16 step of either partner, then one rounding
        assert ((x.double() - y).abs() <= (t + t.roll(64, -1)) * 2 * ULP + y.abs() * ULP).all()
        assert ((x.double() - y).abs() <= y.abs() * ULP + 1e-30).double().mean() > 0.98


@pytest.mark.parametrize("tokens", [1, 9, 800])
def test_qk_norm_rope_without_one_kind_of_heads(lib, tokens):
    """no key heads (or no query heads) and null pointers in their place: the other kind's rows are those of the full call"""
    n, eps = 5, 1e-6
    q, k, qw, kw = rnd(20, tokens, n, 128), rnd(21, tokens, n, 128), rnd(22, 128), rnd(23, 128)
    cos, sin = rnd(24, tokens, 128), rnd(25, tokens, 128)
    a, b, c, d = q.clone(), k.clone(), q.clone(), k.clone()
    lib.prefill_qk_norm_rope_only_cuda(a.data_ptr(), b.data_ptr(), qw.data_ptr(), kw.data_ptr(), cos.data_ptr(), sin.data_ptr(), n, n, 128, tokens, 0, eps, None)
    lib.prefill_qk_norm_rope_only_cuda(c.data_ptr(), None, qw.data_ptr(), None, cos.data_ptr(), sin.data_ptr(), n, 0, 128, tokens, 0, eps, None)
    lib.prefill_qk_norm_rope_only_cuda(None, d.data_ptr(), None, kw.data_ptr(), cos.data_ptr(), sin.data_ptr(), 0, n, 128, tokens, 0, eps, None)
    torch.cuda.synchronize()
    assert torch.equal(a, c) and torch.equal(b, d)


@pytest.mark.parametrize("shift", [0, 4])
@pytest.mark.parametrize("C", [8, 1032, 20])
@pytest.mark.parametrize("T", [1, 2, 3, 15, 16, 17, 50])
def test_conv(lib, T, C, shift):
    x, w, st = rnd(8, T, C, shift=shift), rnd(9, C, 4, scale=0.5), rnd(10, C, 3)
    out, state = torch.zeros(T + 1, C, device="cuda").bfloat16(), st.clone()
    lib.conv1d_prefill_cuda(x.data_ptr(), w.data_ptr(), state.data_ptr(), out.data_ptr(), C, T, 4, None)
    torch.cuda.synchronize()
    full = torch.cat([st.T, x]).double()
    s = sum(full[i:i + T] * w[:, i].double() for i in range(4))
    size = sum((full[i:i + T] * w[:, i].double()).abs() for i in range(4))
    y = s * torch.sigmoid(s)
    # the sum is rounded to bf16 before the activation (slope below 1.1), the result once more
    assert ((out[:T].double() - y).abs() <= 1.1 * (s.abs() * ULP + size * 2 ** -21) + y.abs() * ULP).all()
    assert torch.equal(state, full[-3:].T.bfloat16()) and (out[T] == 0).all()


@pytest.mark.parametrize("T", [262140, 262145, 1048581])
def test_conv_of_many_tokens(lib, T):
    """more blocks of four tokens than the second axis of a grid has places"""
    test_conv(lib, T, 8, 0)


@pytest.mark.parametrize("shift", [0, 4])
@pytest.mark.parametrize("heads,dim", [(1, 128), (15, 128), (16, 128), (33, 128), (7, 96)])
def test_gated_norm(lib, heads, dim, shift):
    x, g = rnd(11, heads, dim, shift=shift), rnd(12, heads, dim)
    w, out = torch.randn(dim, device="cuda"), torch.zeros(heads + 1, dim, device="cuda").bfloat16()
    lib.rms_norm_gated_cuda(x.data_ptr(), w.data_ptr(), g.data_ptr(), out.data_ptr(), heads, dim, 1e-6, None)
    torch.cuda.synchronize()
    d = x.double()
    near(out[:heads], d * torch.rsqrt(d.square().mean(-1, keepdim=True) + 1e-6) * w.double() * g.double() * torch.sigmoid(g.double()), 1.01)
    assert (out[heads] == 0).all()
