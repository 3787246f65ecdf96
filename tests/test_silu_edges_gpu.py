"""x times its logistic in the hybrid layer's kernels: every bf16 argument of the convolution's activation, and gates where the logistic leaves fp32's range."""
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


def test_activation_of_every_bf16(lib):
    """the second of two tokens, 65536 channels, of whose taps the last is 1: the four-tap kernel gives the bits of the three-tap one, which divides with one rounding"""
    C = 1 << 16
    x = torch.zeros(2, C, dtype=BF16, device="cuda")
    x[1] = torch.arange(C, dtype=torch.int32, device="cuda").to(torch.int16).view(BF16)
    got = []
    for taps in (3, 4):
        w = torch.zeros(C, taps, dtype=BF16, device="cuda")
        w[:, -1] = 1
        state, out = torch.zeros(C, taps - 1, dtype=BF16, device="cuda"), torch.zeros_like(x)
        lib.conv1d_prefill_cuda(x.data_ptr(), w.data_ptr(), state.data_ptr(), out.data_ptr(), C, 2, taps, None)
        got.append(out[1])
    torch.cuda.synchronize()
    nan = [g.isnan() for g in got]
    assert torch.equal(nan[0], nan[1])
    assert torch.equal(got[0].view(torch.int16)[~nan[0]], got[1].view(torch.int16)[~nan[1]])


def test_gates_far_below_zero(lib):
    """between -88.7 and -87.3 the logistic is less than 2^-126, and its product with the gate still a normal bf16 value"""
    gate = torch.arange(-88.5, -60.0, 0.5, device="cuda").to(BF16)
    n = gate.numel()
    g = torch.Generator(device="cuda").manual_seed(1)
    x, w = torch.randn(n, 128, generator=g, device="cuda").to(BF16), torch.rand(128, generator=g, device="cuda") + 1
    gates, out = gate[:, None].expand(n, 128).contiguous(), torch.zeros(n, 128, dtype=BF16, device="cuda")
    lib.rms_norm_gated_cuda(x.data_ptr(), w.data_ptr(), gates.data_ptr(), out.data_ptr(), n, 128, 1e-6, None)
    torch.cuda.synchronize()
    v, z = x.to(F64), gates.to(F64)
    want = v * torch.rsqrt(v.square().mean(-1, keepdim=True) + 1e-6) * w.to(F64) * (z / (1 + torch.exp(-z)))
    # one rounding to bf16 of a value that fp32 holds to 1e-6 (expf's own 2 ulp among it), with the spacing of bf16's smallest normal values
    assert ((out.to(F64) - want).abs() <= want.abs() * (2 ** -8 + 1e-5) + 2.0 ** -133).all()
