"""The CTA-pair GEMM (csrc/gemm2.cu) at every tile width that its plan may choose (test_abi.py holds the shapes to that): tokens and features around the tiles, K with a ragged last
block, outputs split at odd places, gated and plain."""
import ctypes as C

import pytest
import torch

from pegainfer_b200 import ffi

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib():
    l = ffi.lib()
    l.cuda_set_device(0)
    l.cublas_init()
    return l


def operands(M, N, K):
    g = torch.Generator(device="cuda").manual_seed(M + 7 * N + K)
    return (torch.randn(M, K, generator=g, device="cuda").mul_(0.1).bfloat16(), torch.randn(N, K, generator=g, device="cuda").bfloat16())


def check(got, W, X):
    """one bf16 rounding (2^-8 relative) of a sum of fp32 products whose K additions round a partial sum of at most |W||X| by 2^-24 each, 64 of them
    at the most in one direction"""
    want, size = X.double() @ W.double().T, X.double().abs() @ W.double().abs().T
    assert ((got.double() - want).abs() <= want.abs() * 2 ** -8 + size * (64 * 2 ** -24)).all()


@pytest.mark.parametrize("M", [15000, 19456, 20001])
@pytest.mark.parametrize("N", [129, 255, 256, 257, 400, 513, 700, 1000])
@pytest.mark.parametrize("K", [264])
def test_against_64_bits(lib, M, N, K):
    W, X = operands(M, N, K)
    Y = torch.full((N + 1, M), 7.0, device="cuda").bfloat16()
    lib.gemm_cuda(W.data_ptr(), X.data_ptr(), Y.data_ptr(), M, N, K, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    check(Y[:N], W, X)
    assert (Y[N] == 7.0).all()


@pytest.mark.parametrize("M,N", [(320, 2100), (480, 2100), (2560, 1000), (2560, 1500), (2560, 2048), (6144, 400), (6144, 1000), (4096, 1500), (1001, 2049)])
def test_every_width(lib, M, N):
    K, e0, e1 = 200, M // 2 + 5, M // 2 + 40
    W, X = operands(M, N, K)
    outs = [torch.zeros(N, w, device="cuda").bfloat16() for w in (e0, e1 - e0, M - e1)]
    rc = lib.pk_b200_gemm_segments(W.data_ptr(), X.data_ptr(), (C.c_void_p * 3)(*[o.data_ptr() for o in outs]), (C.c_int * 3)(e0, e1 - e0, M - e1), M, N, K,
                                   torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert rc == 0
    check(torch.cat(outs, 1), W, X)


@pytest.mark.parametrize("N", [129, 160, 400, 700, 1000, 1300])
@pytest.mark.parametrize("M", [1000, 4099, 9728])
def test_gated(lib, M, N):
    """silu(gate) * up of bf16-rounded products: two roundings more, and silu' is at most 1.1"""
    K = 264
    W, X = operands(2 * M, N, K)
    Y = torch.zeros(N, M, device="cuda").bfloat16()
    assert lib.pk_b200_gemm_swiglu(W.data_ptr(), X.data_ptr(), Y.data_ptr(), M, N, K, torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    p = X.double() @ W.double().T
    g, u = p[:, :M], p[:, M:]
    want = g * torch.sigmoid(g) * u
    bound = 2 ** -8 * (1.1 * g.abs() * u.abs() + 2 * want.abs()) + 2 ** -12
    assert ((Y.double() - want).abs() <= bound * 1.01).all()
