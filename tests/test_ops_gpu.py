"""Op-level parity on the GPU, through the C ABI: every hot-path kernel against the CPU oracle on
the same seeded inputs.  Each case runs twice: on libpegainfer_kernels_b200.so (the product) and,
when oracle/_ref was built, on the reference's own CUDA kernels behind the same ABI -- the second
run is what pins the oracle to the reference on real hardware.

Tolerances (bf16 ulps at max(|want|, floor)): copies and adds are bit-exact; norm / SiLU / RoPE
1-2 ulp (rsqrt.approx, expf, FMA contraction); GEMV / GEMM 1 ulp above a floor of max|y|/64
(fp32 reduction order is unspecified in cuBLAS too); attention 2-3 ulp (ex2.approx, order).
"""
import math
import os

import numpy as np
import pytest
import torch

from oracle import qwen3_oracle as O
from pegainfer_b200 import ffi
from pegainfer_b200.paged_kv import PagedKvLayout
from tests.helpers import assert_bf16_close, bits, from_bits, f32

pytestmark = pytest.mark.gpu

REF_LIB = os.path.join(os.path.dirname(__file__), "..", "oracle", "_ref", "libkernels_ref.so")
LIBS = ["b200"] + (["ref"] if os.path.exists(REF_LIB) else [])
_loaded = {}


def get_lib(kind):
    if kind not in _loaded:
        if kind == "b200":
            lib = ffi.lib()
        else:
            lib = ffi.load(REF_LIB, extensions=False)
        torch.cuda.init()
        torch.zeros(1, device="cuda")
        lib.cuda_set_device(0)
        lib.cublas_init()
        _loaded[kind] = lib
    return _loaded[kind]


@pytest.fixture(params=LIBS)
def lib(request):
    return get_lib(request.param)


def rnd(shape, seed, scale=1.0):
    g = torch.Generator().manual_seed(seed)
    return (torch.randn(shape, generator=g) * scale).to(torch.bfloat16)


_keep = []  # device tensors must outlive the launches that read them (raw pointers cross the ABI)


@pytest.fixture(autouse=True)
def _keepalive():
    _keep.clear()
    yield
    torch.cuda.synchronize()
    _keep.clear()


def dev(t):
    d = t.cuda().contiguous()
    _keep.append(d)
    return d


def p(t):
    return None if t is None else t.data_ptr()


def stream():
    return torch.cuda.current_stream().cuda_stream


def i32(a):
    d = torch.tensor(np.asarray(a, dtype=np.int32), device="cuda")
    _keep.append(d)
    return d


# ------------------------------------------------------------------ embedding / elementwise
@pytest.mark.parametrize("hidden,seq", [(4, 2), (2560, 1), (2560, 37), (260, 3)])
def test_embedding(lib, hidden, seq):
    vocab = 97
    embed = rnd((vocab, hidden), 1)
    ids = torch.randint(0, vocab, (seq,), generator=torch.Generator().manual_seed(2), dtype=torch.int32)
    out = torch.zeros((seq, hidden), dtype=torch.bfloat16, device="cuda")
    e_d, ids_d = dev(embed), dev(ids)
    rc = lib.embedding_batched_cuda(p(e_d), p(ids_d), p(out), hidden, seq, stream())
    assert rc == 0
    want = O.embedding_batched(bits(embed), ids.numpy().astype(np.uint32), hidden)
    assert (bits(out) == want).all()
    out1 = torch.zeros(hidden, dtype=torch.bfloat16, device="cuda")
    assert lib.embedding_decode_cuda(p(e_d), p(ids_d), p(out1), hidden, stream()) == 0
    assert (bits(out1) == want[0]).all()


def test_embedding_vocab_shard(lib):  # pegainfer-kernels/src/ops/embedding.rs:99-128
    embed = from_bits(O.f32_to_bf16(np.array([10, 11, 12, 20, 21, 22], np.float32))).reshape(2, 3)
    ids = dev(torch.tensor([4, 5, 1, 4], dtype=torch.int32))
    out = torch.zeros((4, 3), dtype=torch.bfloat16, device="cuda")
    assert lib.embedding_batched_vocab_shard_cuda(p(dev(embed)), p(ids), p(out), 3, 4, 4, 2, stream()) == 0
    assert out.float().cpu().flatten().tolist() == [10, 11, 12, 20, 21, 22, 0, 0, 0, 10, 11, 12]


@pytest.mark.parametrize("n", [5, 2560, 2560 * 33 + 3])
def test_add(lib, n):
    a, b = rnd((n,), 3), rnd((n,), 4)
    out = torch.zeros(n, dtype=torch.bfloat16, device="cuda")
    assert lib.add_cuda(p(dev(a)), p(dev(b)), p(out), n, stream()) == 0
    assert (bits(out) == O.add(bits(a), bits(b))).all()


@pytest.mark.parametrize("inter,bs", [(9728, 1), (9728, 5), (52, 3)])
def test_silu_mul_fused(lib, inter, bs):
    gu = rnd((bs, 2 * inter), 5, 2.0)
    out = torch.zeros((bs, inter), dtype=torch.bfloat16, device="cuda")
    lib.silu_mul_fused_cuda(p(dev(gu)), p(out), inter, bs, stream())
    assert_bf16_close(bits(out), O.silu_mul_fused(bits(gu), inter), 1, floor=1e-3, frac_exact=0.98,
                      what="silu_mul_fused")


def test_silu_mul_rounded(lib):
    g, u = rnd((4096,), 6, 2.0), rnd((4096,), 7)
    out = torch.zeros(4096, dtype=torch.bfloat16, device="cuda")
    assert lib.silu_mul_triton_aot_cuda(p(dev(g)), p(dev(u)), p(out), 4096, stream()) == 0
    assert_bf16_close(bits(out), O.silu_mul(bits(g), bits(u)), 1, floor=1e-3, frac_exact=0.98)


# ------------------------------------------------------------------ norms
@pytest.mark.parametrize("hidden,seq", [(4, 1), (260, 2), (2560, 1), (2560, 19), (4096, 4)])
def test_rms_norm(lib, hidden, seq):
    x, w = rnd((seq, hidden), 8, 3.0), rnd((hidden,), 9, 0.2) + 1
    out = torch.zeros_like(x, device="cuda")
    lib.rms_norm_batched_cuda(p(dev(x)), p(dev(w)), p(out), hidden, seq, 1e-6, stream())
    assert_bf16_close(bits(out), O.rms_norm(bits(x), bits(w), 1e-6), 1, frac_exact=0.97, what="rms_norm")
    if seq == 1:
        out1 = torch.zeros_like(x, device="cuda")
        lib.rms_norm_cuda(p(dev(x)), p(dev(w)), p(out1), hidden, 1e-6, stream())
        assert (bits(out1) == bits(out)).all()


def test_rms_norm_reference_known_answers(lib):  # ops/tests.rs:88-152
    x = from_bits(O.f32_to_bf16(np.array([1, 2, 3, 4], np.float32)))
    w = from_bits(O.f32_to_bf16(np.ones(4, np.float32)))
    out = torch.zeros(4, dtype=torch.bfloat16, device="cuda")
    lib.rms_norm_cuda(p(dev(x)), p(dev(w)), p(out), 4, 1e-6, stream())
    inv = 1.0 / math.sqrt((1 + 4 + 9 + 16) / 4 + 1e-6)
    assert np.abs(out.float().cpu().numpy() - np.array([1, 2, 3, 4]) * inv).max() <= 0.01


@pytest.mark.parametrize("hidden,bs", [(2560, 1), (2560, 7), (4096, 2), (260, 3)])
def test_fused_add_rms_norm(lib, hidden, bs):
    h, r, w = rnd((bs, hidden), 10, 2.0), rnd((bs, hidden), 11, 0.5), rnd((hidden,), 12, 0.2) + 1
    h_d, out = dev(h), torch.zeros((bs, hidden), dtype=torch.bfloat16, device="cuda")
    lib.fused_add_rms_norm_batched_cuda(p(h_d), p(dev(r)), p(dev(w)), p(out), hidden, bs, 1e-6, stream())
    h_np = bits(h).copy()
    want = O.fused_add_rms_norm(h_np, bits(r), bits(w), 1e-6)
    assert (bits(h_d) == h_np).all(), "hidden += residual must be bit-exact"
    assert_bf16_close(bits(out), want, 1, frac_exact=0.97, what="fused_add_rms_norm")


# ------------------------------------------------------------------ GEMV / GEMM
def test_gemv_known_answer(lib):  # ops/tests.rs:50-77
    a = from_bits(O.f32_to_bf16(np.array([1, 2, 3, 4, 5, 6], np.float32))).reshape(2, 3)
    x = from_bits(O.f32_to_bf16(np.array([1, 2, 3], np.float32)))
    y = torch.zeros(2, dtype=torch.bfloat16, device="cuda")
    lib.gemm_graphsafe_cuda(p(dev(a)), p(dev(x)), p(y), 2, 1, 3, stream())
    assert y.float().cpu().tolist() == [14.0, 32.0]


@pytest.mark.parametrize("M,K", [(1024, 2560), (2560, 9728), (6144, 2560), (151936 // 8, 2560), (333, 1288)])
def test_gemv_stream(lib, M, K):
    W, x = rnd((M, K), 13, 0.02), rnd((1, K), 14, 1.0)
    y = torch.zeros((1, M), dtype=torch.bfloat16, device="cuda")
    lib.gemm_graphsafe_cuda(p(dev(W)), p(dev(x)), p(y), M, 1, K, stream())
    want = O.gemm(bits(W), bits(x))
    floor = float(np.abs(f32(want)).max()) / 64
    assert_bf16_close(bits(y), want, 1, floor=floor, frac_exact=0.9, what=f"gemv {M}x{K}")


@pytest.mark.parametrize("N", [2, 3, 4])
def test_gemv_multi_token(lib, N):
    M, K = 2048, 2560
    W, x = rnd((M, K), 15, 0.02), rnd((N, K), 16, 1.0)
    y = torch.zeros((N, M), dtype=torch.bfloat16, device="cuda")
    lib.gemm_graphsafe_cuda(p(dev(W)), p(dev(x)), p(y), M, N, K, stream())
    want = O.gemm(bits(W), bits(x))
    assert_bf16_close(bits(y), want, 1, floor=float(np.abs(f32(want)).max()) / 64, frac_exact=0.9)


@pytest.mark.parametrize("M,N,K", [(512, 128, 2560), (2560, 77, 4096), (1000, 130, 576), (4096, 300, 2560),
                                   (19456, 128, 2560), (64, 8, 64), (24, 16, 40),
                                   # CTA-pair kernel (N > 128): full + ragged token / feature tiles, several K depths
                                   (2560, 512, 4096), (6144, 257, 2560), (2560, 1024, 9728), (136, 129, 64), (19456, 2048, 2560),
                                   # 320-wide pair tiles (two 160-column accumulators): one wave for 2560 features at 2048 tokens
                                   (2560, 2048, 1024), (2400, 2047, 320)])
def test_gemm(lib, M, N, K):
    W, X = rnd((M, K), 17, 0.02), rnd((N, K), 18, 1.0)
    Y = torch.zeros((N, M), dtype=torch.bfloat16, device="cuda")
    lib.gemm_cuda(p(dev(W)), p(dev(X)), p(Y), M, N, K, stream())
    torch.cuda.synchronize()
    want = O.gemm(bits(W), bits(X))
    assert_bf16_close(bits(Y), want, 1, floor=float(np.abs(f32(want)).max()) / 64, frac_exact=0.9,
                      what=f"gemm {M}x{N}x{K}")


@pytest.mark.parametrize("inter,N,K", [(9728, 512, 2560), (1000, 300, 576), (128, 129, 64)])
def test_gemm_swiglu_epilogue(inter, N, K):
    """gate_up GEMM with SwiGLU in the epilogue == gemm + silu_mul_fused (oracle composition, prefill.rs:168-176)."""
    lib = get_lib("b200")
    W, X = rnd((2 * inter, K), 27, 0.03), rnd((N, K), 28, 1.0)
    act = torch.zeros((N, inter), dtype=torch.bfloat16, device="cuda")
    rc = lib.pk_b200_gemm_swiglu(p(dev(W)), p(dev(X)), p(act), inter, N, K, stream())
    assert rc == 0
    torch.cuda.synchronize()
    want = O.silu_mul_fused(O.gemm(bits(W), bits(X)), inter)
    # gate and up are each within 1 ulp of the oracle after their bf16 rounding; silu(g) * u compounds them
    assert_bf16_close(bits(act), want, 3, floor=float(np.abs(f32(want)).max()) / 64, frac_exact=0.85, what=f"gemm+swiglu {inter}x{N}x{K}")
    # one token tile is not a pair problem: the entry says so and the caller falls back
    assert lib.pk_b200_gemm_swiglu(p(dev(W)), p(dev(X)), p(act), inter, 64, K, stream()) == -2


@pytest.mark.parametrize("M,N,K", [(2560, 8, 2560), (2560, 64, 9728), (1024, 33, 2560)])
def test_gemm_graphsafe_batch_bucket(lib, M, N, K):  # decode bucket > 4 goes to the tensor-core path (gemm_skinny.cu)
    W, X = rnd((M, K), 19, 0.02), rnd((N, K), 20, 1.0)
    W_d, X_d = dev(W), dev(X)
    Y = torch.zeros((N, M), dtype=torch.bfloat16, device="cuda")
    lib.gemm_graphsafe_cuda(p(W_d), p(X_d), p(Y), M, N, K, stream())
    want = O.gemm(bits(W), bits(X))
    assert_bf16_close(bits(Y), want, 1, floor=float(np.abs(f32(want)).max()) / 64, frac_exact=0.9)
    # the parts of K are added up in a fixed order: repeated launches are bit-identical
    Y2 = torch.zeros_like(Y)
    for _ in range(3):
        lib.gemm_graphsafe_cuda(p(W_d), p(X_d), p(Y2), M, N, K, stream())
    torch.cuda.synchronize()
    assert (bits(Y2) == bits(Y)).all()


# ------------------------------------------------------------------ QK norm + RoPE
@pytest.mark.parametrize("tokens,nq,nkv,decode", [(1, 32, 8, True), (5, 32, 8, True), (37, 32, 8, False), (3, 4, 1, True)])
def test_qk_norm_rope(lib, tokens, nq, nkv, decode):
    hd = 128
    q, k = rnd((tokens, nq * hd), 21, 2.0), rnd((tokens, nkv * hd), 22, 2.0)
    qw, kw = rnd((hd,), 23, 0.3) + 1, rnd((hd,), 24, 0.3) + 1
    cos, sin = O.precompute_rope(hd, 4096, 1e6)
    q_d, k_d = dev(q), dev(k)
    cos_d, sin_d = from_bits(cos, "cuda"), from_bits(sin, "cuda")
    qn, kn = bits(q).copy(), bits(k).copy()
    if decode:
        pos = np.array([(17 * i + 3) % 4096 for i in range(tokens)], np.int32)
        lib.qk_norm_rope_batched_decode_cuda(p(q_d), p(k_d), p(dev(qw)), p(dev(kw)), p(cos_d), p(sin_d),
                                             p(i32(pos)), nq, nkv, hd, tokens, 1e-6, stream())
        O.qk_norm_rope(qn, kn, bits(qw), bits(kw), cos, sin, nq, nkv, hd, 1e-6, positions=pos)
    else:
        lib.prefill_qk_norm_rope_only_cuda(p(q_d), p(k_d), p(dev(qw)), p(dev(kw)), p(cos_d), p(sin_d),
                                           nq, nkv, hd, tokens, 11, 1e-6, stream())
        O.qk_norm_rope(qn, kn, bits(qw), bits(kw), cos, sin, nq, nkv, hd, 1e-6, start_pos=11)
    assert_bf16_close(bits(q_d), qn, 2, floor=2 ** -6, frac_exact=0.9, what="q rope")
    assert_bf16_close(bits(k_d), kn, 2, floor=2 ** -6, frac_exact=0.9, what="k rope")


# ------------------------------------------------------------------ paged KV + attention
class Paged:
    """Synthetic paged pool for one layer-agnostic test: L layers, shuffled page ids."""

    def __init__(self, seq_lens, nkv, num_layers=2, seed=0, fill=True):
        self.layout = PagedKvLayout.new(num_layers, nkv, 128, 16)
        rng = np.random.RandomState(seed)
        need = [-(-s // 16) for s in seq_lens]
        total = sum(need) + 3
        ids = rng.permutation(np.arange(1, total + 1))
        self.page_indices, self.indptr, self.last = [], [0], []
        off = 0
        for s, n in zip(seq_lens, need):
            self.page_indices += ids[off:off + n].tolist()
            off += n
            self.indptr.append(len(self.page_indices))
            self.last.append(((s - 1) % 16) + 1 if s else 0)
        self.num_pages = total + 1
        g = torch.Generator().manual_seed(seed + 100)
        n_el = self.num_pages * self.layout.page_stride
        self.kv = (torch.randn(n_el, generator=g) * (1.0 if fill else 0.0)).to(torch.bfloat16)
        self.pi = np.array(self.page_indices, np.int32)
        self.ip = np.array(self.indptr, np.int32)
        self.lpl = np.array(self.last, np.int32)


@pytest.mark.parametrize("nkv", [8, 1])
def test_paged_kv_scatter(lib, nkv):
    hd, seq_lens, layer = 128, [40, 7, 16], 1
    pg = Paged(seq_lens, nkv, fill=False)
    L = pg.layout
    toks = [(b, t) for b, s in enumerate(seq_lens) for t in range(s) if (t * 7 + b) % 3 != 0]
    bidx = np.array([b for b, _ in toks], np.int32)
    pos = np.array([t for _, t in toks], np.int32)
    k, v = rnd((len(toks), nkv * hd), 30), rnd((len(toks), nkv * hd), 31)
    kv_d = dev(pg.kv)
    rc = lib.paged_kv_scatter_cuda(p(kv_d), L.k_offset(layer), L.v_offset(layer), p(i32(pg.pi)), p(i32(pg.ip)),
                                   p(i32(pg.lpl)), p(dev(k)), p(dev(v)), p(i32(bidx)), p(i32(pos)), len(toks),
                                   nkv, hd, 16, L.page_stride, nkv * hd, hd, stream())
    assert rc == 0
    want = bits(pg.kv).copy()
    O.paged_kv_scatter(want, L.k_offset(layer), L.v_offset(layer), pg.pi, pg.ip, pg.lpl, bits(k), bits(v),
                       bidx, pos, nkv, hd, 16, L.page_stride)
    assert (bits(kv_d) == want).all()


@pytest.mark.parametrize("seq_lens,nq,nkv", [([1], 32, 8), ([128], 32, 8), ([191, 33, 1], 32, 8), ([700], 4, 1),
                                             ([1500, 900], 32, 8), ([4090], 32, 8), ([3000, 17, 640], 32, 8),
                                             ([100, 260, 16, 15, 17], 32, 8), ([4096], 8, 2), ([300, 3000], 16, 4)])
def test_paged_attention_decode(lib, seq_lens, nq, nkv):
    hd, layer, bs = 128, 1, len(seq_lens)
    pg = Paged(seq_lens, nkv, seed=3)
    L = pg.layout
    q = rnd((bs, nq * hd), 32)
    out = torch.zeros((bs, nq * hd), dtype=torch.bfloat16, device="cuda")
    req, tile0, chunk = np.arange(bs, dtype=np.int32), np.zeros(bs, np.int32), np.array(seq_lens, np.int32)
    sm = 1 / math.sqrt(hd)
    rc = lib.paged_attention_decode_cuda(p(dev(q)), p(out), p(dev(pg.kv)), L.k_offset(layer), L.v_offset(layer),
                                         p(i32(pg.pi)), p(i32(pg.ip)), p(i32(pg.lpl)), p(i32(req)), p(i32(tile0)),
                                         p(i32(chunk)), nq, nkv, hd, 16, bs, L.page_stride, sm, stream())
    assert rc == 0
    want = O.paged_attention_decode(bits(q), bits(pg.kv), L.k_offset(layer), L.v_offset(layer), pg.pi, pg.ip,
                                    pg.lpl, req, tile0, chunk, nq, nkv, hd, 16, L.page_stride, sm)
    assert_bf16_close(bits(out), want, 3, floor=float(np.abs(f32(want)).max()) / 32, what="decode attn")


@pytest.mark.parametrize("dirty", ["latent", "grouped"])
def test_paged_attention_decode_behind_other_splits(dirty):
    """The counters of the split decode attention live in the thread's scratch memory and have to be zero: kernels that leave partial sums of their own there in
    between must not touch them (they did, and outputs stayed unwritten)."""
    lib = get_lib("b200")
    bf = lambda *s: (1 + torch.rand(*s, device="cuda")).bfloat16()  # noqa: E731
    n, H = 3000, 20
    pages, zero, pos = i32(np.arange(n // 16 + 1, dtype=np.int32)), i32(np.zeros(1, np.int32)), i32(np.array([n - 1], np.int32))
    if dirty == "latent":
        q, cache, out = bf(H, 192), bf(n // 16 + 1, 16, 192), bf(H, 128)
        assert lib.pk_latent_attention_ex(p(q), p(cache), None, p(pos), p(zero), p(zero), p(pages), p(out), 16 * 192, 16, 1, H, 128, 64, 0.07, 0, n, 0, stream()) == 0
    else:  # over 16 heads to a group: tiles of 64 rows with the keys dealt out
        q, cache, out = bf(H, 128), bf(n // 16 + 1, 16, 256), bf(H, 128)
        ex = ffi.AttnExtra(window=0, softcap=0.0, slope_log2=0.0, keep_first=0, gate=None, gate_ld=0, gate_per_head=0, max_kv_len=n)
        import ctypes as C
        assert lib.pk_gqa_attention_ex(p(q), p(cache), None, p(pos), p(zero), p(zero), p(pages), p(out), 16 * 256, 16, 1, H, 1, 128, 128, 0.09, 0, C.byref(ex), 0,
                                       stream()) == 0
    torch.cuda.synchronize()
    test_paged_attention_decode(lib, [3000, 17, 640], 16, 8)


@pytest.mark.parametrize("seq_lens", [[1024], [2300, 1100]])
def test_paged_attention_decode_split_kv(lib, seq_lens):
    nq, nkv, hd, layer, bs = 32, 8, 128, 0, len(seq_lens)
    pg = Paged(seq_lens, nkv, seed=4)
    L = pg.layout
    q = rnd((bs, nq * hd), 33)
    csz = max(256, -(-max(seq_lens) // 64))
    sreq, stile, mask, oip = [], [], [], [0]
    for b, s in enumerate(seq_lens):
        n = max(1, -(-s // csz))
        sreq += [b] * n; stile += list(range(n)); mask += [1] * n; oip.append(len(sreq))
    pad = bs * 64 - len(sreq)
    sreq += [0] * pad; stile += [0] * pad; mask += [0] * pad
    sreq, stile = np.array(sreq, np.int32), np.array(stile, np.int32)
    mask, oip, csz_a = np.array(mask, np.uint8), np.array(oip, np.int32), np.array([csz], np.int32)
    slots = len(sreq)
    out = torch.zeros((bs, nq * hd), dtype=torch.bfloat16, device="cuda")
    tmp_v = torch.zeros((slots, nq * hd), dtype=torch.bfloat16, device="cuda")
    tmp_s = torch.zeros((slots, nq), dtype=torch.float32, device="cuda")
    sm = 1 / math.sqrt(hd)
    rc = lib.paged_attention_decode_split_kv_cuda(
        p(dev(q)), p(out), p(dev(pg.kv)), L.k_offset(layer), L.v_offset(layer), p(i32(pg.pi)), p(i32(pg.ip)),
        p(i32(pg.lpl)), p(i32(sreq)), p(i32(stile)), p(i32(csz_a)), p(i32(oip)),
        p(dev(torch.tensor(mask))), p(tmp_v), p(tmp_s), nq, nkv, hd, 16, bs, slots, L.page_stride, sm,
        stream())
    assert rc == 0
    want = O.paged_attention_decode_split_kv(bits(q), bits(pg.kv), L.k_offset(layer), L.v_offset(layer), pg.pi,
                                             pg.ip, pg.lpl, sreq, stile, csz_a, oip, mask, nq, nkv, hd, 16, bs,
                                             L.page_stride, sm)
    assert_bf16_close(bits(out), want, 5, floor=float(np.abs(f32(want)).max()) / 32, what="split-kv attn")


@pytest.mark.parametrize("starts,lens,nq,nkv", [([0], [128], 32, 8), ([0], [77], 32, 8), ([0, 0, 0], [33, 100, 5], 32, 8),
                                                ([40], [60], 32, 8), ([0], [300], 4, 1)])
def test_batch_prefill_paged(lib, starts, lens, nq, nkv):
    hd, layer, bs = 128, 1, len(lens)
    kv_lens = [s + n for s, n in zip(starts, lens)]
    pg = Paged(kv_lens, nkv, seed=5)
    L = pg.layout
    T = sum(lens)
    q = rnd((T, nq * hd), 34)
    out = torch.zeros((T, nq * hd), dtype=torch.bfloat16, device="cuda")
    q_indptr = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    group = nq // nkv
    tile_q = lib.batch_prefill_cta_tile_q_with_override(T, nq, nkv, hd, 64)
    assert tile_q == 64
    ri, qti = [], []
    for b, n in enumerate(lens):
        for t in range(-(-n * group // tile_q)):
            ri.append(b); qti.append(t)
    nt = len(ri)
    sm = 1 / math.sqrt(hd)
    rc = lib.batch_prefill_paged_cuda_with_cta_tile_q(
        p(dev(q)), p(out), p(dev(pg.kv)), L.k_offset(layer), L.v_offset(layer), p(i32(pg.pi)), p(i32(pg.ip)),
        p(i32(pg.lpl)), p(i32(q_indptr)), p(i32(ri)), p(i32(qti)), p(i32(np.zeros(nt))), p(i32(kv_lens)),
        p(i32([T])), nq, nkv, hd, 16, T, bs, nt, L.page_stride, sm, 64,
        stream())
    assert rc == 0
    want = O.batch_prefill_paged(bits(q), bits(pg.kv), L.k_offset(layer), L.v_offset(layer), pg.pi, pg.ip, pg.lpl,
                                 q_indptr, nq, nkv, hd, 16, L.page_stride, sm)
    # P is rounded to bf16 against the RUNNING row max in the kernels (ours and FA2) and against the final
    # max in the oracle: uncorrelated 2^-9 roundings -> a few ulp at the max/32 floor
    assert_bf16_close(bits(out), want, 8, floor=float(np.abs(f32(want)).max()) / 32, what="prefill attn")


def test_prefill_planner_helpers(lib):  # csrc/paged_attention.cu:343-397
    assert lib.batch_prefill_cta_tile_q(2048, 32, 8, 128) == 128
    assert lib.batch_prefill_cta_tile_q(8, 32, 8, 128) == 64
    assert lib.batch_prefill_cta_tile_q(2, 32, 8, 128) == 16
    assert lib.batch_prefill_cta_tile_q_with_override(2048, 32, 8, 128, 64) == 64
    assert lib.batch_prefill_cta_tile_q_with_override(2048, 32, 8, 128, 48) == 0
    assert lib.batch_prefill_paged_num_tiles_with_cta_tile_q(2048, 32, 8, 128, 64) == 128
    assert lib.batch_prefill_paged_num_tiles_with_cta_tile_q(2048, 32, 8, 128, 48) == -1
    assert lib.batch_prefill_paged_num_tiles(100, 32, 8, 128) == 4


# ------------------------------------------------------------------ sampling
def test_argmax_known_answer(lib):  # ops/tests.rs:79-86
    x = from_bits(O.f32_to_bf16(np.array([1.0, 9.0, 3.0, 8.0], np.float32)), "cuda")
    out = torch.zeros(1, dtype=torch.int32, device="cuda")
    lib.argmax_cuda(p(x), p(out), 4, stream())
    assert int(out.item()) == 1


@pytest.mark.parametrize("n", [5, 1000, 151936])
def test_top1_matches_argmax(lib, n):
    x = rnd((n,), 40, 3.0)
    want = O.argmax(bits(x))
    xf = x.float()
    out = torch.zeros(1, dtype=torch.int32, device="cuda")
    lib.argmax_cuda(p(dev(x)), p(out), n, stream())
    assert int(out.item()) == want  # argmax.cu:18: lowest index wins ties
    val = torch.zeros(8, dtype=torch.bfloat16, device="cuda")
    states = torch.zeros(1 << 20, dtype=torch.uint8, device="cuda")
    for _ in range(2):  # twice: the scratch must be left reusable
        out.zero_()
        lib.flashinfer_top1_cuda(p(dev(x)), p(val), p(states), p(out), n, stream())
        got = int(out.item())
        assert float(xf[got]) == float(xf[want])  # the reference's radix top-1 leaves tie ORDER undefined
        if lib is get_lib("b200"):
            assert got == want  # ours: lowest index
            # ours also returns the winner's VALUE (both the multi-CTA and the small-row path): the vocab-sharded
            # tensor-parallel top-1 exchange compares it across ranks
            assert float(val[0].float()) == float(xf[want])


# ------------------------------------------------------------------ non-greedy sampling
def _sample(lib, logits, inv_t, top_k, top_p, seed):
    n = logits.numel()
    probs = torch.zeros(n, dtype=torch.float32, device="cuda")
    valid = torch.zeros(8, dtype=torch.uint8, device="cuda")
    out = torch.full((1,), -1, dtype=torch.int32, device="cuda")
    lib.gpu_sample_flashinfer_cuda(p(logits), p(probs), p(valid), p(out), n, inv_t, top_k, top_p, seed, stream())
    torch.cuda.synchronize()
    return int(out.item()), probs


def test_gpu_sample_reference_cases(lib):  # pegainfer-server/src/ops/tests.rs:228-305
    logits = dev(from_bits(O.f32_to_bf16(np.array([1.0, 2.0, 10.0, 1.5, 0.5], np.float32))))
    tok, _ = _sample(lib, logits, 1.0 / 0.01, -1, 1.0, 0x3f000000)  # near-greedy
    assert tok == 2
    tok, _ = _sample(lib, logits, 1.0, -1, 1.0, 0)  # plain temperature sampling stays in range
    assert 0 <= tok < 5
    tok, _ = _sample(lib, logits, 1.0, 1, 1.0, 0x3f000000)  # top_k = 1
    assert tok == 2


def test_gpu_sample_distribution_and_filters():
    """Ours only (the random stream is ours): softmax probs exact to fp32, top-k / top-p never leave the
    eligible set, and the empirical distribution over 3000 seeds matches the renormalised probabilities."""
    lib = get_lib("b200")
    g = torch.Generator().manual_seed(7)
    logits_h = (torch.randn(64, generator=g) * 2).to(torch.bfloat16)
    logits = dev(logits_h)
    pr = torch.softmax(logits_h.float() * 0.8, dim=0).numpy().astype(np.float64)
    _, probs = _sample(lib, logits, 0.8, -1, 1.0, 1)
    assert np.abs(probs.cpu().numpy() - pr).max() < 1e-6
    order = np.argsort(-pr)
    topk = set(order[:5].tolist())
    cum = np.cumsum(pr[order])
    nucleus = set(order[:int(np.searchsorted(cum, 0.6) + 1)].tolist())
    counts = np.zeros(64)
    for seed in range(3000):
        tok, _ = _sample(lib, logits, 0.8, 5, 1.0, seed)
        assert tok in topk
        counts[tok] += 1
        if seed < 300:
            assert _sample(lib, logits, 0.8, -1, 0.6, seed)[0] in nucleus
            assert _sample(lib, logits, 0.8, 5, 0.6, seed)[0] in (topk & nucleus)
    want = np.array([pr[i] if i in topk else 0.0 for i in range(64)])
    want /= want.sum()
    sigma = np.sqrt(3000 * want * (1 - want)) + 1
    assert (np.abs(counts - 3000 * want) <= 5 * sigma).all()
    # vocabulary-sized call: in range, greedy-equivalent with top_k = 1
    big = dev(rnd((151936,), 41, 3.0))
    # top_k = 1 keeps every token tied at the maximum; the pick must be one of them
    top = _sample(lib, big, 1.0, 1, 1.0, 5)[0]
    assert float(big[top]) == float(big.float().max())
    tok, _ = _sample(lib, big, 1.0, 50, 0.9, 123)
    assert 0 <= tok < 151936


# ------------------------------------------------------------------ B200 extensions, op level (ours only)
def test_gemm_segments_matches_three_gemms():
    lib = get_lib("b200")
    import ctypes as C
    qd, kd, H, T = 4096, 1024, 2560, 200
    W, X = rnd((qd + 2 * kd, H), 50, 0.02), rnd((T, H), 51, 1.0)
    W_d, X_d = dev(W), dev(X)
    outs = [torch.zeros((T, n), dtype=torch.bfloat16, device="cuda") for n in (qd, kd, kd)]
    ptrs = (C.c_void_p * 3)(*[o.data_ptr() for o in outs])
    segs = (C.c_int * 3)(qd, kd, kd)
    assert lib.pk_b200_gemm_segments(p(W_d), p(X_d), ptrs, segs, qd + 2 * kd, T, H, stream()) == 0
    row = 0
    for o, n in zip(outs, (qd, kd, kd)):
        ref = torch.zeros((T, n), dtype=torch.bfloat16, device="cuda")
        lib.gemm_cuda(W_d.data_ptr() + row * H * 2, p(X_d), p(ref), n, T, H, stream())
        torch.cuda.synchronize()
        assert (bits(o) == bits(ref)).all()  # same kernel, same tiles along K: bit-identical
        row += n
    want = O.gemm(bits(W[:qd]), bits(X))
    assert_bf16_close(bits(outs[0]), want, 1, floor=float(np.abs(f32(want)).max()) / 64, frac_exact=0.9)


@pytest.mark.parametrize("T", [129, 160, 256, 257, 700])
@pytest.mark.parametrize("segs,H", [((4096, 1024, 1024), 4096), ((512, 128, 128), 2560), ((512, 64, 64), 4096), ((4096, 1024, 1024), 5120), ((1000, 64, 300), 8184)])
def test_gemm_segments_are_the_single_calls_bit_for_bit(segs, H, T):
    """what the header promises from 129 tokens on: hidden widths around and above 4096, one key / value head of a shard, odd sizes"""
    lib = get_lib("b200")
    import ctypes as C
    g = torch.Generator(device="cuda").manual_seed(H + T)
    W = torch.randn(sum(segs), H, generator=g, device="cuda").mul_(0.02).bfloat16()
    X = torch.randn(T, H, generator=g, device="cuda").bfloat16()
    outs = [torch.zeros((T, n), dtype=torch.bfloat16, device="cuda") for n in segs]
    assert lib.pk_b200_gemm_segments(p(W), p(X), (C.c_void_p * 3)(*[o.data_ptr() for o in outs]), (C.c_int * 3)(*segs), sum(segs), T, H, stream()) == 0
    row = 0
    for o, n in zip(outs, segs):
        ref = torch.zeros((T, n), dtype=torch.bfloat16, device="cuda")
        lib.gemm_cuda(W.data_ptr() + row * H * 2, p(X), p(ref), n, T, H, stream())
        torch.cuda.synchronize()
        assert torch.equal(o, ref)
        row += n


@pytest.mark.parametrize("N", [1, 3])
def test_gemv_fused_prologue_epilogue(N):
    """x_mode 1 (residual add + RMSNorm prologue) with three output segments, then epi 1 (SwiGLU)."""
    lib = get_lib("b200")
    import ctypes as C
    H, qd, kd, inter = 2560, 4096, 1024, 9728
    hid, res, nw = rnd((N, H), 60, 1.0), rnd((N, H), 61, 0.3), rnd((H,), 62, 0.2) + 1
    W = rnd((qd + 2 * kd, H), 63, 0.02)
    outs = [torch.zeros((N, n), dtype=torch.bfloat16, device="cuda") for n in (qd, kd, kd)]
    hout = torch.zeros((N, H), dtype=torch.bfloat16, device="cuda")
    g = ffi.GemvArgs()
    g.W, g.X = p(dev(W)), p(dev(hid))
    g.Y = (C.c_void_p * 3)(*[o.data_ptr() for o in outs])
    g.seg_rows = (C.c_int * 3)(qd, kd, kd)
    g.M, g.N, g.K, g.x_mode = qd + 2 * kd, N, H, 1
    g.residual, g.norm_w, g.eps, g.hidden_out, g.normed_out, g.epi = p(dev(res)), p(dev(nw)), 1e-6, p(hout), None, 0
    assert lib.pk_b200_gemv_fused(C.byref(g), stream()) == 0
    h_np = bits(hid).copy()
    normed = O.fused_add_rms_norm(h_np, bits(res), bits(nw), 1e-6)
    assert (bits(hout) == h_np).all()
    want = O.gemm(bits(W), normed)
    got = np.concatenate([bits(o) for o in outs], axis=1)
    assert_bf16_close(got, want, 2, floor=float(np.abs(f32(want)).max()) / 64, frac_exact=0.85, what="fused qkv gemv")
    # SwiGLU epilogue on a gate|up matrix
    Wgu, x = rnd((2 * inter, H), 64, 0.02), rnd((N, H), 65, 1.0)
    act = torch.zeros((N, inter), dtype=torch.bfloat16, device="cuda")
    g2 = ffi.GemvArgs()
    g2.W, g2.X = p(dev(Wgu)), p(dev(x))
    g2.Y = (C.c_void_p * 3)(act.data_ptr(), None, None)
    g2.seg_rows = (C.c_int * 3)(inter, 0, 0)
    g2.M, g2.N, g2.K, g2.x_mode, g2.epi = inter, N, H, 0, 1
    assert lib.pk_b200_gemv_fused(C.byref(g2), stream()) == 0
    want = O.silu_mul_fused(O.gemm(bits(Wgu), bits(x)), inter)
    assert_bf16_close(bits(act), want, 2, floor=float(np.abs(f32(want)).max()) / 64, frac_exact=0.85, what="swiglu gemv")


# ------------------------------------------------------------------ fused decode attention (+ L2 prefetch clusters)
@pytest.mark.parametrize("seq_lens", [[1], [300], [2300, 77], [4095], [17, 2049, 512, 16]])
def test_decode_attention_fused_matches_unfused_ops(seq_lens):
    """pk_b200_decode_attention_fused == qk_norm_rope_batched_decode + paged_kv_scatter + paged_attention_decode
    (oracle composition, batch_decode.rs:196-247), and the prefetch variant returns the same bits."""
    lib = get_lib("b200")
    nq, nkv, hd, layer, bs = 32, 8, 128, 1, len(seq_lens)
    pg = Paged(seq_lens, nkv, seed=9)
    L = pg.layout
    q, k, v = rnd((bs, nq * hd), 40, 2.0), rnd((bs, nkv * hd), 41, 2.0), rnd((bs, nkv * hd), 42)
    qw, kw = rnd((hd,), 43, 0.3) + 1, rnd((hd,), 44, 0.3) + 1
    cos, sin = O.precompute_rope(hd, 4096, 1e6)
    pos = np.array([s - 1 for s in seq_lens], np.int32)
    sm = 1 / math.sqrt(hd)
    # oracle: norm+rope -> append -> attention over the full context
    qn, kn = bits(q).copy(), bits(k).copy()
    O.qk_norm_rope(qn, kn, bits(qw), bits(kw), cos, sin, nq, nkv, hd, 1e-6, positions=pos)
    kv_want = bits(pg.kv).copy()
    O.paged_kv_scatter(kv_want, L.k_offset(layer), L.v_offset(layer), pg.pi, pg.ip, pg.lpl, kn, bits(v),
                       np.arange(bs, dtype=np.int32), pos, nkv, hd, 16, L.page_stride)
    req, tile0, chunk = np.arange(bs, dtype=np.int32), np.zeros(bs, np.int32), np.array(seq_lens, np.int32)
    want = O.paged_attention_decode(qn, kv_want, L.k_offset(layer), L.v_offset(layer), pg.pi, pg.ip, pg.lpl, req, tile0,
                                    chunk, nq, nkv, hd, 16, L.page_stride, sm)
    max_chunks = 37
    cos_d, sin_d = from_bits(cos, "cuda"), from_bits(sin, "cuda")
    _keep.extend([cos_d, sin_d])
    weights = rnd((4096, 2560), 45)  # stands in for the next GEMVs' weights
    w_d = dev(weights)
    spans = (ffi.PrefetchSpan * 2)(ffi.PrefetchSpan(p(w_d), 4096, 5120, lib.pk_b200_gemv_grid(4096, 0), 64),
                                   ffi.PrefetchSpan(p(w_d), 2048, 5120, lib.pk_b200_gemv_grid(2048, 1), 3))
    outs = []
    for use_pf in (False, True):
        kv_d = dev(pg.kv)
        out = torch.zeros((bs, nq * hd), dtype=torch.bfloat16, device="cuda")
        partial = torch.zeros(bs * max_chunks * nq * 130, dtype=torch.float32, device="cuda")
        counters = torch.zeros(bs * nkv + 16, dtype=torch.int32, device="cuda")
        common = [p(dev(q)), p(dev(k)), p(dev(v)), p(out), p(kv_d), L.k_offset(layer), L.v_offset(layer), p(i32(pg.pi)),
                  p(i32(pg.ip)), p(i32(pg.lpl)), p(i32(pos)), p(dev(qw)), p(dev(kw)), p(cos_d), p(sin_d), 1e-6, p(partial), p(counters), 64, max_chunks, nq, nkv, hd, 16, bs,
                  L.page_stride, sm]
        _keep.extend([partial, counters])
        if use_pf:
            rc = lib.pk_b200_decode_attention_fused_prefetch(*common, spans, 2, stream())
        else:
            rc = lib.pk_b200_decode_attention_fused(*common, stream())
        assert rc == 0
        torch.cuda.synchronize()
        assert_bf16_close(bits(out), want, 3, floor=float(np.abs(f32(want)).max()) / 32, what="fused decode attn")
        # the appended K/V rows are the oracle's bits (norm/rope within 2 ulp -> compare through the attention only),
        # V rows are plain copies
        got_kv = bits(kv_d)
        vmask = got_kv != bits(pg.kv)
        assert vmask.sum() <= bs * 2 * nkv * hd
        outs.append(bits(out).copy())
    assert (outs[0] == outs[1]).all(), "prefetch clusters must not change the result"


def test_decode_attention_prefetch_rejects_bad_spans():
    lib = get_lib("b200")
    assert lib.pk_b200_gemv_grid(2560, 0) == min(2 * torch.cuda.get_device_properties(0).multi_processor_count, 320)
    assert lib.pk_b200_gemv_grid(16, 1) == 4
    bad = (ffi.PrefetchSpan * 1)(ffi.PrefetchSpan(16, 8, 24, 4, 1))  # row_bytes % 16 != 0
    z = torch.zeros(4096, dtype=torch.bfloat16, device="cuda")
    zi = torch.zeros(64, dtype=torch.int32, device="cuda")
    rc = lib.pk_b200_decode_attention_fused_prefetch(p(z), p(z), p(z), p(z), p(z), 0, 0, p(zi), p(zi), p(zi), p(zi), p(z), p(z),
                                                     p(z), p(z), 1e-6, None, p(zi), 64, 1, 32, 8, 128, 16, 1, 32768, 0.1, bad, 1,
                                                     stream())
    assert rc == -1


# ------------------------------------------------------------------ tcgen05 prefill attention (direct entry)
@pytest.mark.parametrize("impl", ["tc2", "tc"])
@pytest.mark.parametrize("starts,lens,nq,nkv", [([0], [128], 32, 8), ([0, 0, 0], [33, 100, 5], 32, 8), ([40], [60], 32, 8),
                                                ([0], [300], 4, 1), ([100, 0], [700, 129], 32, 8), ([0], [256], 8, 2),
                                                ([0], [257], 8, 2), ([900], [300], 8, 2), ([0], [1536], 4, 1),
                                                ([0, 3, 250], [1, 130, 390], 8, 2)])
def test_prefill_attention_tc(starts, lens, nq, nkv, impl, monkeypatch):
    """The tcgen05/TMEM flash-attention kernels (TMA page loads, MN-major V operand; tc2 = two query tiles per CTA with O
    and P in tensor memory, the default; tc = one tile per CTA) against the oracle, same tolerance as the mma.sync
    kernel behind the ABI entry (test_batch_prefill_paged).  Cases cover a single tile, a tile pair with the second
    tile short by one / long by one token, chunked prefill (causal offset 900), 12 KV blocks, and a ragged batch."""
    monkeypatch.setenv("PK_PREFILL_ATTN", impl)
    lib = get_lib("b200")
    hd, layer, bs = 128, 1, len(lens)
    kv_lens = [s + n for s, n in zip(starts, lens)]
    pg = Paged(kv_lens, nkv, seed=6)
    L = pg.layout
    T = sum(lens)
    q = rnd((T, nq * hd), 35)
    out = torch.zeros((T, nq * hd), dtype=torch.bfloat16, device="cuda")
    q_indptr = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    sm = 1 / math.sqrt(hd)
    rc = lib.pk_b200_prefill_attention_tc(p(dev(q)), p(out), p(dev(pg.kv)), L.k_offset(layer), L.v_offset(layer),
                                          p(i32(pg.pi)), p(i32(pg.ip)), p(i32(pg.lpl)), p(i32(q_indptr)), nq, nkv, hd, 16, T,
                                          bs, L.page_stride, sm, stream())
    assert rc == 0
    want = O.batch_prefill_paged(bits(q), bits(pg.kv), L.k_offset(layer), L.v_offset(layer), pg.pi, pg.ip, pg.lpl,
                                 q_indptr, nq, nkv, hd, 16, L.page_stride, sm)
    from tests.helpers import ulp_err
    e = ulp_err(bits(out).ravel(), np.asarray(want).ravel(), float(np.abs(f32(want)).max()) / 32)
    print(f"\n[prefill attention {impl}] lens {lens} starts {starts}: max err {e.max():.2f} ulp, {float((e == 0).mean()):.4f} bit-exact")
    # Measured on B200: 1.1-2.5 ulp on every case but the one whose chunk starts
    # 900 tokens into the request (6.7 ulp): there the kernels' 128-token blocks and the oracle's 64-token tiles advance the
    # running maximum at different KV positions over a long cached prefix, so more P values round differently.
    tol = 8 if max(starts) >= 512 else 4
    assert_bf16_close(bits(out), want, tol, floor=float(np.abs(f32(want)).max()) / 32, what="tc prefill attn")
    assert lib.pk_b200_prefill_attention_tc(p(dev(q)), p(out), p(dev(pg.kv)), L.k_offset(layer), L.v_offset(layer),
                                            p(i32(pg.pi)), p(i32(pg.ip)), p(i32(pg.lpl)), p(i32(q_indptr)), nq, nkv, hd, 32,
                                            T, bs, L.page_stride, sm, stream()) == -1  # page size 32: unsupported


@pytest.mark.parametrize("start,n", [(0, 1), (0, 80), (0, 96), (0, 97), (0, 112), (0, 113), (128, 95), (128, 96), (128, 97), (30, 200), (0, 352)])
def test_prefill_attention_parts_of_p(start, n):
    """Key counts around the six of eight 16-key steps of a block after which P V begins; against float64.  P and the result are each
    rounded to bf16 (2^-9 relative at most) and the sum's denominator is that of the rounded P: 2^-8 in the norm, with room for fp32."""
    lib = get_lib("b200")
    nq, nkv, hd, layer = 8, 2, 128, 1
    pg = Paged([start + n], nkv, seed=n)
    L = pg.layout
    q = rnd((n, nq * hd), n + 1)
    out = torch.zeros((n, nq * hd), dtype=torch.bfloat16, device="cuda")
    assert lib.pk_b200_prefill_attention_tc(p(dev(q)), p(out), p(dev(pg.kv)), L.k_offset(layer), L.v_offset(layer), p(i32(pg.pi)), p(i32(pg.ip)),
                                            p(i32(pg.lpl)), p(i32(np.array([0, n], np.int32))), nq, nkv, hd, 16, n, 1, L.page_stride, 1 / math.sqrt(hd), stream()) == 0
    kv = pg.kv.double()
    def rows(off):
        pages = [kv[off + int(i) * L.page_stride:][:16 * nkv * hd].view(16, nkv, hd) for i in pg.pi]
        return torch.cat(pages)[:start + n].transpose(0, 1).repeat_interleave(nq // nkv, 0)
    K, V = rows(L.k_offset(layer)), rows(L.v_offset(layer))
    Q = q.double().cpu().view(n, nq, hd).transpose(0, 1)
    s = Q @ K.transpose(1, 2) / math.sqrt(hd)
    s.masked_fill_(torch.ones(n, start + n, dtype=torch.bool).triu(start + 1), -math.inf)
    want = (s.softmax(-1) @ V).transpose(0, 1).reshape(n, -1)
    got = out.cpu().double()
    assert (got - want).norm() <= 2.0 ** -8 * want.norm()


# ------------------------------------------------------------------ tensor-parallel collectives, the peer's lines laid down on ONE GPU
# Kernels that wait for one another never run side by side on one GPU: the ranks run one after the other, and what the first one waits for lies in its
# staging buffer before it is launched.  So no wait goes round more than once.
STAGING = 1 << 20
SLOT = (STAGING // 4) & ~15  # bytes of a (slot, source) region of a world of two; its last eighth holds the lines
LINES = SLOT - (SLOT // 8 & ~15)


def _two_ranks(lib):
    """Communicators of a world of two whose staging and flag buffers all lie on this GPU (the 'NVLink' writes are local)"""
    import ctypes as C
    stage = [torch.zeros(STAGING, dtype=torch.uint8, device="cuda") for _ in range(2)]
    flags = [torch.zeros(int(lib.pk_tp_flag_bytes()), dtype=torch.uint8, device="cuda") for _ in range(2)]
    sp = (C.c_void_p * 2)(stage[0].data_ptr(), stage[1].data_ptr())
    fp = (C.c_void_p * 2)(flags[0].data_ptr(), flags[1].data_ptr())
    comms = [lib.pk_tp_comm_create(r, 2, sp, fp, STAGING) for r in range(2)]
    assert all(comms) and all(lib.pk_tp_set_wait_limit(c, 1000) == 0 for c in comms)  # (a line in the wrong place ends as a test that fails)
    _keep.extend(stage + flags)
    return comms, [s.view(torch.int32) for s in stage]


@pytest.mark.parametrize("N", [1, 3])
def test_gemv_ll_allreduce_with_the_peers_lines(N):
    """epi 3: GEMV + all-reduce of the CTA's own rows in one kernel.  Each 'rank' holds a column slice of W and the
    matching slice of x (row-parallel o_proj / down_proj); both must write the rank-ordered bf16 sum of the two bf16
    partials, bit-identical to the oracle's all-reduce model, for consecutive ops (slot / sequence reuse)."""
    lib = get_lib("b200")
    import ctypes as C
    M, K = 512, 1024
    comms, stage = _two_ranks(lib)
    step = torch.tensor([7], dtype=torch.int32, device="cuda")
    for op in range(3):
        W, x = rnd((M, 2 * K), 70 + op, 0.05), rnd((N, 2 * K), 80 + op, 1.0)
        parts, outs, own, args = [], [], [], []
        for r in range(2):
            Wr = dev(W[:, r * K:(r + 1) * K].contiguous())
            xr = dev(x[:, r * K:(r + 1) * K].contiguous())
            y, partial = (torch.zeros((N, M), dtype=torch.bfloat16, device="cuda") for _ in range(2))
            g = ffi.GemvArgs()
            g.W, g.X = p(Wr), p(xr)
            g.Y = (C.c_void_p * 3)(partial.data_ptr(), None, None)
            g.seg_rows = (C.c_int * 3)(M, 0, 0)
            g.M, g.N, g.K, g.x_mode, g.epi = M, N, K, 0, 0
            assert lib.pk_b200_gemv_fused(C.byref(g), stream()) == 0  # the rank's partial rows
            g.Y = (C.c_void_p * 3)(y.data_ptr(), None, None)
            g.epi, g.tp_comm, g.tp_step, g.tp_op = 3, comms[r], step.data_ptr(), op
            args.append(g)
            outs.append(y)
            own.append(partial)
            parts.append(O.gemm(bits(W[:, r * K:(r + 1) * K].contiguous()), bits(x[:, r * K:(r + 1) * K].contiguous())))
        # a line per pair of tokens and row: two bf16 values, the sequence number
        pairs = torch.zeros(((N + 1) // 2, M, 2), dtype=torch.bfloat16, device="cuda")
        for n in range(N):
            pairs[n // 2, :, n % 2] = own[1][n]
        lines = torch.stack([pairs.view(torch.int32)[..., 0], torch.full((pairs.shape[0], M), 7 * 256 + op + 1, dtype=torch.int32, device="cuda")], -1).flatten()
        at = (((op & 1) * 2 + 1) * SLOT + LINES) // 4  # rank 1's region in rank 0's buffer
        here = stage[0][at:at + lines.numel()]
        here.copy_(lines)
        torch.cuda.synchronize()
        assert lib.pk_b200_gemv_fused(C.byref(args[0]), stream()) == 0
        torch.cuda.synchronize()
        here.zero_()
        torch.cuda.synchronize()
        assert lib.pk_b200_gemv_fused(C.byref(args[1]), stream()) == 0  # finds what rank 0's kernel left
        torch.cuda.synchronize()
        assert lib.pk_b200_wait_errors() == 0 and torch.equal(here, lines)  # and leaves the lines that were laid down before
        want = O.all_reduce_sum(parts)
        assert (bits(outs[0]) == bits(outs[1])).all(), "ranks disagree"
        assert_bf16_close(bits(outs[0]), want, 2, floor=float(np.abs(f32(want)).max()) / 64, frac_exact=0.85, what=f"ll all-reduce op {op}")


def test_tp_top1_exchange_with_the_peers_lines():
    """Vocab-sharded greedy token: every rank ends with the same global (max, lowest index) winner."""
    lib = get_lib("b200")
    comms, stage = _two_ranks(lib)
    step = torch.tensor([3], dtype=torch.int32, device="cuda")

    def exchange(vals, local, step, op, seq, entry):
        idx = [torch.tensor(i, dtype=torch.int32, device="cuda") for i in local]
        v = [from_bits(O.f32_to_bf16(np.array(x, np.float32)), "cuda") for x in vals]
        n = len(vals[0])
        seq -= 1 << 32 if seq >> 31 else 0
        lines = torch.stack([v[1].float().view(torch.int32), torch.full_like(idx[1], seq), idx[1] + 1000, torch.full_like(idx[1], seq)], 1).flatten()
        at = (2 * SLOT - 4096 + entry * 16) // 4  # rank 1's region in rank 0's buffer
        here = stage[0][at:at + 4 * n]
        here.copy_(lines)
        for r in range(2):
            torch.cuda.synchronize()
            assert lib.pk_tp_top1_exchange(comms[r], p(v[r]), p(idx[r]), n, r * 1000, step.data_ptr() if step is not None else None, op, stream()) == 0
            torch.cuda.synchronize()
            if r == 0:
                here.zero_()
        assert lib.pk_b200_wait_errors() == 0 and torch.equal(here, lines)
        assert idx[0].tolist() == idx[1].tolist()
        return idx[0].tolist()

    # request 0: rank 1 wins (4.0 at 1000+5); request 1: tie at 9.0 -> lowest global index (rank 0: 20); request 2: rank 0 (30)
    vals = ([1.5, 9.0, 2.0], [4.0, 9.0, -1.0])
    assert exchange(vals, ([10, 20, 30], [5, 6, 7]), step, 250, 3 * 256 + 251, 0) == [1005, 20, 30]
    # host-path sequence numbers (no step counter) use separate lines
    assert exchange(([1.5], [4.0]), ([3], [4]), None, 0x80000001, 0x80000001, 64) == [1004]
