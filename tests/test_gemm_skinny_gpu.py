"""The few-tile GEMM (csrc/gemm_skinny.cu) behind gemm_cuda / pk_b200_gemm_segments at the sizes where it can go wrong: token counts around its
tile widths, feature counts around its tiles, K with a ragged last block and too short to cut, outputs split at odd places, unaligned rows."""
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


def check(got, W, X):
    """one bf16 rounding (2^-8 relative) of a sum of fp32 products: each of the K additions rounds a partial sum of at most |W||X| by 2^-24, and
    they are spread over several partials, so 64 such roundings bound what is seen"""
    want, size = X.double() @ W.double().T, X.double().abs() @ W.double().abs().T
    assert ((got.double() - want).abs() <= want.abs() * 2 ** -8 + size * (64 * 2 ** -24)).all()


@pytest.mark.parametrize("pdl", [0, 1])
@pytest.mark.parametrize("N", [5, 16, 17, 32, 33, 48, 49, 64, 65, 96, 97, 128, 129, 160, 257])
@pytest.mark.parametrize("M,K", [(32, 2560), (40, 72), (136, 8), (2560, 4096), (6144, 264), (1001, 1032), (12, 520)])
def test_against_64_bits(lib, M, K, N, pdl):
    g = torch.Generator(device="cuda").manual_seed(M + 7 * N + K)
    W = torch.randn(M, K, generator=g, device="cuda").mul_(0.1).bfloat16()
    X = torch.randn(N, K, generator=g, device="cuda").bfloat16()
    Y = torch.full((N + 1, M), 7.0, device="cuda").bfloat16()
    lib.pk_b200_set_pdl(pdl)
    try:
        for _ in range(2):  # the second launch behind the first
            lib.gemm_cuda(W.data_ptr(), X.data_ptr(), Y.data_ptr(), M, N, K, torch.cuda.current_stream().cuda_stream)
    finally:
        lib.pk_b200_set_pdl(0)
    torch.cuda.synchronize()
    check(Y[:N], W, X)
    assert (Y[N] == 7.0).all() and lib.pk_b200_wait_errors() == 0


@pytest.mark.parametrize("N", [6, 100, 131])
@pytest.mark.parametrize("segs", [(64, 32, 32), (70, 3, 55), (8, 0, 250), (1, 2, 300), (4096, 1024, 1024)])
def test_three_outputs(lib, segs, N):
    M, K = sum(segs), 520
    g = torch.Generator(device="cuda").manual_seed(M + N)
    W = torch.randn(M, K, generator=g, device="cuda").mul_(0.1).bfloat16()
    X = torch.randn(N, K, generator=g, device="cuda").bfloat16()
    outs = [torch.zeros(N, max(s, 1), device="cuda").bfloat16() for s in segs]
    rc = lib.pk_b200_gemm_segments(W.data_ptr(), X.data_ptr(), (C.c_void_p * 3)(*[o.data_ptr() for o in outs]), (C.c_int * 3)(*segs), M, N, K,
                                   torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    torch.cuda.synchronize()
    check(torch.cat([o for o, s in zip(outs, segs) if s], 1), W, X)


@pytest.mark.parametrize("N,M,K", [(64, 4096, 2560), (128, 2560, 512), (200, 1024, 4096)])
def test_product_as_the_weights_of_a_gemv(lib, N, M, K):
    """The kernel for one row streams its weights before it waits for its predecessor: a product that is used as weights has to be complete by then."""
    g = torch.Generator(device="cuda").manual_seed(N)
    W = [torch.randn(M, K, generator=g, device="cuda").mul_(0.1).bfloat16() for _ in range(4)]
    X = torch.randn(N, K, generator=g, device="cuda").bfloat16()
    v = torch.randn(M, generator=g, device="cuda").bfloat16()
    Y, out = torch.zeros(N, M, device="cuda").bfloat16(), torch.zeros(len(W), N, device="cuda").bfloat16()
    st = torch.cuda.current_stream().cuda_stream
    lib.pk_b200_set_pdl(1)
    try:
        for i, w in enumerate(W):
            lib.gemm_cuda(w.data_ptr(), X.data_ptr(), Y.data_ptr(), M, N, K, st)
            lib.gemm_cuda(Y.data_ptr(), v.data_ptr(), out[i].data_ptr(), N, 1, M, st)
    finally:
        lib.pk_b200_set_pdl(0)
    torch.cuda.synchronize()
    check(Y, W[-1], X)
    for i, w in enumerate(W):  # the products of this run, rounded once
        lib.gemm_cuda(w.data_ptr(), X.data_ptr(), Y.data_ptr(), M, N, K, st)
        torch.cuda.synchronize()
        check(out[i:i + 1], Y, v[None])
