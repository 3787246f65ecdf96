"""Tensor-parallel products of 2 to 4 tokens (gemv.cu): rows reduced inside the kernel (epilogue 3) and rows pushed to the peers (epilogue 2) with the prologue that
sums them (x_mode 2).  Odd numbers of rows, several blocks of row pairs in a CTA.  Two ranks on one GPU, one after the other: a rank finds in its buffers what
it waits for, the peer's lines laid down before, or the peer's push already made."""
import ctypes as C

import pytest
import torch

from pegainfer_b200 import ffi

pytestmark = pytest.mark.gpu
BF16, I32 = torch.bfloat16, torch.int32
STAGING = 4 << 20
SLOT = (STAGING // 4) & ~15                # bytes of a (parity, source) region of a world of two
LINES = SLOT - (SLOT // 8 & ~15)           # where its lines begin
CTL = 2 * 64 * 8                           # word of the flags with the sequence number; before it, per parity, 64 x 8 flags


@pytest.fixture(scope="module")
def lib():
    l = ffi.lib()
    l.cuda_set_device(0)
    l.cublas_init()
    return l


def two_ranks(lib):
    stage = [torch.zeros(STAGING, dtype=torch.uint8, device="cuda") for _ in range(2)]
    flags = [torch.zeros(int(lib.pk_tp_flag_bytes()), dtype=torch.uint8, device="cuda") for _ in range(2)]
    at = [(C.c_void_p * 2)(*[t.data_ptr() for t in ts]) for ts in (stage, flags)]
    comms = [lib.pk_tp_comm_create(r, 2, *at, STAGING) for r in range(2)]
    assert all(comms) and all(lib.pk_tp_set_wait_limit(c, 1000) == 0 for c in comms)
    return comms, stage, flags


def gemv(lib, W, X, Y, N, epi, **more):
    a = ffi.GemvArgs()
    a.W, a.X, a.M, a.N, a.K, a.epi = W.data_ptr(), X.data_ptr(), W.shape[0], N, W.shape[1], epi
    a.Y[0], a.seg_rows[0] = Y.data_ptr(), W.shape[0]
    for k, v in more.items():
        setattr(a, k, v.data_ptr() if isinstance(v, torch.Tensor) else v)
    return lib.pk_b200_gemv_fused(C.byref(a), None)


def parts(lib, N, M, K):
    """each rank's weights, activations and plain result"""
    g = torch.Generator(device="cuda").manual_seed(M + N)
    rn = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    W, X = [(rn(M, K) * K ** -0.5).to(BF16) for _ in range(2)], [rn(N, K).to(BF16) for _ in range(2)]
    Y = [torch.zeros(N, M, dtype=BF16, device="cuda") for _ in range(2)]
    for w, x, y in zip(W, X, Y):
        assert gemv(lib, w, x, y, N, 0) == 0
    return W, X, Y


SHAPES = [(513, 1024), (1, 520), (296, 2048), (6501, 12288)]  # the last: two blocks of row pairs in a CTA


@pytest.mark.parametrize("N", [2, 3, 4])
@pytest.mark.parametrize("M,K", SHAPES)
def test_reduced_inside(lib, N, M, K):
    comms, stage, flags = two_ranks(lib)
    step = torch.tensor([5], dtype=I32, device="cuda")
    for op in range(2):
        W, X, own = parts(lib, N, M, K)
        pairs = torch.zeros((N + 1) // 2, M, 2, dtype=BF16, device="cuda")  # a line per pair of tokens and row: two values, the sequence number
        for n in range(N):
            pairs[n // 2, :, n % 2] = own[1][n]
        lines = torch.stack([pairs.view(I32)[..., 0], torch.full((pairs.shape[0], M), 5 * 256 + op + 1, dtype=I32, device="cuda")], -1).flatten()
        at = (((op & 1) * 2 + 1) * SLOT + LINES) // 4  # rank 1's region in rank 0's buffer
        here = stage[0].view(I32)[at:at + lines.numel()]
        here.copy_(lines)
        out = [torch.full((N, M), float("nan"), dtype=BF16, device="cuda") for _ in range(2)]
        for r in range(2):
            torch.cuda.synchronize()
            assert gemv(lib, W[r], X[r], out[r], N, 3, tp_comm=comms[r], tp_step=step, tp_op=op) == 0
            torch.cuda.synchronize()
            if r == 0:
                here.zero_()
        assert lib.pk_b200_wait_errors() == 0 and torch.equal(here, lines)
        want = (own[0].float() + own[1].float()).to(BF16)  # two terms: one rounding whatever the order
        assert torch.equal(out[0], want) and torch.equal(out[1], want)


@pytest.mark.parametrize("N", [2, 3, 4])
@pytest.mark.parametrize("M,K", SHAPES)
def test_pushed_and_summed_by_the_next(lib, N, M, K):
    comms, stage, flags = two_ranks(lib)
    words = [f.view(I32) for f in flags]
    for seq in (1, 2):
        W, X, own = parts(lib, N, M, K)
        none = torch.zeros(N, M, dtype=BF16, device="cuda")
        for r in range(2):
            assert gemv(lib, W[r], X[r], none, N, 2, tp_comm=comms[r]) == 0
            torch.cuda.synchronize()
        for to in range(2):
            assert words[to][CTL].item() == seq and words[to][CTL + 2].item() == 0
            for src in range(2):
                assert words[to][(seq & 1) * 64 * 8 + src].item() == seq
                at = ((seq & 1) * 2 + src) * SLOT
                assert torch.equal(stage[to][at:at + N * M * 2].view(BF16).view(N, M), own[src])
        if M % 8 or M > 10240:
            continue
        g = torch.Generator(device="cuda").manual_seed(M)
        rn = lambda *s: torch.randn(*s, generator=g, device="cuda").to(BF16)  # noqa: E731
        V, hidden, nw = (rn(300, M).float() * M ** -0.5).to(BF16), rn(N, M), rn(M)
        y, h, x = torch.zeros(N, 300, dtype=BF16, device="cuda"), torch.zeros_like(hidden), torch.zeros_like(hidden)
        assert gemv(lib, V, hidden, y, N, 0, x_mode=2, norm_w=nw, eps=1e-6, hidden_out=h, normed_out=x, tp_comm=comms[seq % 2]) == 0
        torch.cuda.synchronize()
        s = hidden.double() + (own[0].float() + own[1].float()).to(BF16).double()
        n = s * torch.rsqrt(s.square().mean(-1, keepdim=True) + 1e-6) * nw.double()
        assert torch.equal(h, s.to(BF16)) and ((x.double() - n).abs() <= n.abs() * (2 ** -8 + 1e-5)).all()
        z = x.double() @ V.double().T
        assert ((y.double() - z).abs() <= z.abs() * 2 ** -8 + 1e-4).all()
    assert lib.pk_b200_wait_errors() == 0


@pytest.mark.parametrize("epi", [2, 3])
def test_more_rows_than_a_cta_keeps_are_refused(lib, epi):
    comms, stage, flags = two_ranks(lib)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    step = torch.zeros(1, dtype=I32, device="cuda")
    x = torch.zeros(2, 64, dtype=BF16, device="cuda")
    W, y = (torch.zeros(128 * sms + 1, k, dtype=BF16, device="cuda") for k in (64, 2))
    before = [t.clone() for t in (*stage, *flags)]
    assert gemv(lib, W, x, y, 2, epi, tp_comm=comms[0], tp_step=step) != 0
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(before, (*stage, *flags)))
