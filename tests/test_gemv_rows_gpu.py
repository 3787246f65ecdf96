"""Products of 2 to 4 tokens (gemv.cu) against 64 bits at the edges: odd numbers of rows, rows of a few elements and of several chunks, the longest
activations, more row pairs than a block's sums hold."""
import ctypes as C

import pytest
import torch

from pegainfer_b200 import ffi

pytestmark = pytest.mark.gpu
BF16, F64 = torch.bfloat16, torch.float64


@pytest.fixture(scope="module")
def lib():
    l = ffi.lib()
    l.cuda_set_device(0)
    l.cublas_init()
    return l


def args(W, X, Ys, rows, M, N, K, **more):
    a = ffi.GemvArgs()
    a.W, a.X, a.M, a.N, a.K = W.data_ptr(), X.data_ptr(), M, N, K
    for i, y in enumerate(Ys):
        a.Y[i], a.seg_rows[i] = y.data_ptr(), rows[i]
    for k, v in more.items():
        setattr(a, k, v.data_ptr() if isinstance(v, torch.Tensor) else v)
    return a


def close(got, want, scale):
    """one rounding to bf16 beside fp32 sums"""
    return ((got.to(F64) - want).abs() <= want.abs() * 2 ** -8 + scale * 1e-5).all()


@pytest.mark.parametrize("N", [2, 3, 4])
@pytest.mark.parametrize("M,K", [(1, 8), (2, 264), (7, 1024), (149, 1032), (295, 2560), (297, 4096), (2560, 9728), (300, 12288), (100001, 64)])
def test_plain(lib, N, M, K):
    g = torch.Generator(device="cuda").manual_seed(M + K + N)
    W, X = torch.randn(M, K, generator=g, device="cuda").to(BF16), torch.randn(N, K, generator=g, device="cuda").to(BF16)
    cut = [M] if M < 7 else [M // 3, M // 2, M - M // 3 - M // 2]
    Ys = [torch.full((N, m), float("nan"), dtype=BF16, device="cuda") for m in cut]
    assert lib.pk_b200_gemv_fused(C.byref(args(W, X, Ys, cut, M, N, K)), None) == 0
    torch.cuda.synchronize()
    assert close(torch.cat(Ys, 1), X.to(F64) @ W.to(F64).T, K ** 0.5)


@pytest.mark.parametrize("N", [2, 3, 4])
@pytest.mark.parametrize("M,K,x_mode,epi", [(1, 64, 1, 1), (151, 2560, 1, 1), (300, 520, 3, 4), (40, 10240, 1, 5), (33, 2048, 0, 6)])
def test_gated(lib, N, M, K, x_mode, epi):
    g = torch.Generator(device="cuda").manual_seed(M + K + N)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda").to(BF16)  # noqa: E731
    W, X, R, nw = (r(2 * M, K).float() * K ** -0.5).to(BF16), r(N, K), r(N, K), r(K)
    Y, H = torch.zeros(N, M, dtype=BF16, device="cuda"), torch.zeros(N, K, dtype=BF16, device="cuda")
    assert lib.pk_b200_gemv_fused(C.byref(args(W, X, [Y], [M], M, N, K, x_mode=x_mode, epi=epi, residual=R, norm_w=nw, eps=1e-6, hidden_out=H)), None) == 0
    torch.cuda.synchronize()
    x = X.to(F64)
    if x_mode:
        h = x + R.to(F64)
        assert torch.equal(H, h.to(BF16))
        if x_mode == 3:
            h = h.to(BF16).to(F64)
        x = (h * torch.rsqrt(h.square().mean(-1, keepdim=True) + 1e-6) * (nw.to(F64) + (1 if x_mode == 3 else 0))).to(BF16).to(F64)
    z = x @ W.to(F64).T
    a, b = z[:, :M].to(BF16).to(F64), z[:, M:].to(BF16).to(F64)
    s = torch.relu(a) if epi == 5 else a * torch.sigmoid(1.5957691216057308 * (a + 0.044715 * a ** 3)) if epi == 6 else a * torch.sigmoid(a)
    # the gate's and the up row's own roundings may fall the other way: 2^-8 of either factor, and one more for the result
    assert ((Y.to(F64) - s * b).abs() <= (s * b).abs() * 2 ** -6 + 0.01 * (b.abs() + s.abs()) * 2 ** -3 + 1e-3).all()
