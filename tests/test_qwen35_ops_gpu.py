"""GPU parity of the Qwen3.5 hybrid-layer ops (pegainfer_b200/csrc/qwen35_ops.cu) against oracle/qwen35_oracle.py.

On a B200 the token-by-token hybrid forward of tests/tools/qwen35_bringup.py matches the oracle within 2.25 ulp at the row max over 24 steps."""
import math
import os

import numpy as np
import pytest
import torch

from oracle import qwen3_oracle as O
from oracle.qwen35_oracle import gated_delta_rule_step, rb, rms_norm_offset, silu
from pegainfer_b200 import ffi
from tests.helpers import assert_bf16_close, bits, f32

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib():
    l = ffi.lib()
    torch.zeros(1, device="cuda")
    l.cuda_set_device(0)
    l.cublas_init()  # the thread workspace: the delta-rule sequence kernel takes its pre-pass version with it
    return l


def rnd(shape, seed, scale=1.0):
    g = torch.Generator().manual_seed(seed)
    return (torch.randn(shape, generator=g) * scale).to(torch.bfloat16)


def st():
    return torch.cuda.current_stream().cuda_stream


def vals(t):  # bf16 tensor -> fp32 numpy of its values
    return f32(bits(t))


def test_rms_norm_offset(lib):
    x, w = rnd((5, 2560), 1, 2.0), rnd((2560,), 2, 0.2)
    xd, wd = x.cuda(), w.cuda()
    out = torch.empty_like(xd)
    lib.rms_norm_batched_offset_cuda(xd.data_ptr(), wd.data_ptr(), out.data_ptr(), 2560, 5, 1e-6, st())
    want = O.f32_to_bf16(rms_norm_offset(vals(x), vals(w), 1e-6))
    assert_bf16_close(bits(out), want, 1, what="rms_norm_offset")


def test_rms_norm_gated(lib):
    nh, hd = 3 * 32, 128  # 3 tokens x 32 value heads, weight broadcast over heads
    x, g = rnd((nh, hd), 3), rnd((nh, hd), 4)
    w = torch.randn(hd, generator=torch.Generator().manual_seed(5)) * 0.3 + 1
    xd, gd, wd = x.cuda(), g.cuda(), w.cuda()
    out = torch.empty_like(xd)
    lib.rms_norm_gated_cuda(xd.data_ptr(), wd.data_ptr(), gd.data_ptr(), out.data_ptr(), nh, hd, 1e-6, st())
    xv, gv = vals(x), vals(g)
    inv = 1.0 / np.sqrt((xv * xv).mean(-1, keepdims=True, dtype=np.float32) + np.float32(1e-6))
    want = O.f32_to_bf16(xv * inv * w.numpy()[None] * silu(gv))
    assert_bf16_close(bits(out), want, 2, floor=2 ** -8, what="rms_norm_gated")


@pytest.mark.parametrize("T", [1, 2, 37])
def test_conv1d_prefill_and_state(lib, T):
    C, K = 8192, 4
    x, w, s0 = rnd((T, C), 6), rnd((C, K), 7, 0.5), rnd((C, K - 1), 8)
    xd, wd, sd = x.cuda(), w.cuda(), s0.cuda()
    out = torch.empty_like(xd)
    lib.conv1d_prefill_cuda(xd.data_ptr(), wd.data_ptr(), sd.data_ptr(), out.data_ptr(), C, T, K, st())
    xv, wv, sv = vals(x), vals(w), vals(s0)
    hist = np.concatenate([sv.T, xv], axis=0)  # [K-1 + T, C], oldest first
    acc = np.zeros((T, C), np.float32)
    for k in range(K):
        acc += hist[k:k + T] * wv[:, k][None]
    want = O.f32_to_bf16(silu(rb(acc)))
    assert_bf16_close(bits(out), want, 2, floor=2 ** -8, what="conv1d+silu")
    assert (bits(sd) == O.f32_to_bf16(hist[-(K - 1):].T)).all(), "conv state = last K-1 inputs"


def test_gated_delta_rule_decode(lib):
    nk, nv, dk, dv = 16, 32, 128, 128
    g = torch.Generator().manual_seed(9)
    qkv = rnd((2 * nk * dk + nv * dv,), 10)
    a, b, dtb = rnd((nv,), 11), rnd((nv,), 12), rnd((nv,), 13, 0.5)
    a_log = torch.randn(nv, generator=g) * 0.5
    S = (torch.randn((nv, dk, dv), generator=g) * 0.1).float()
    Sd = S.cuda()
    out = torch.empty(nv * dv, dtype=torch.bfloat16, device="cuda")
    qkv_d, b_d, a_d, dtb_d, alog_d = qkv.cuda(), b.cuda(), a.cuda(), dtb.cuda(), a_log.cuda()  # keep alive across the launch
    lib.gated_delta_rule_decode_cuda(qkv_d.data_ptr(), b_d.data_ptr(), a_d.data_ptr(), dtb_d.data_ptr(), alog_d.data_ptr(), Sd.data_ptr(),
                                     out.data_ptr(), nk, nv, dk, dv, st())
    torch.cuda.synchronize()
    qv = vals(qkv)
    Sw = S.numpy().copy()
    want = gated_delta_rule_step(qv[:nk * dk].reshape(nk, dk), qv[nk * dk:2 * nk * dk].reshape(nk, dk), qv[2 * nk * dk:].reshape(nv, dv),
                                 vals(a), vals(b), vals(dtb), a_log.numpy(), Sw)
    assert_bf16_close(bits(out), O.f32_to_bf16(want.reshape(-1)), 2, floor=float(np.abs(want).max()) / 64, what="gdr out")
    np.testing.assert_allclose(Sd.cpu().numpy(), Sw, rtol=1e-4, atol=1e-5)


def _norm_rope_ref(h, nw, cos, sin, pos, rd, eps):
    inv = 1.0 / np.sqrt((h * h).mean(-1, keepdims=True, dtype=np.float32) + np.float32(eps))
    n = rb(h * inv * (1.0 + nw))
    lo, hi = n[..., : rd // 2].copy(), n[..., rd // 2: rd].copy()
    c, s = cos[pos, : rd // 2], sin[pos, : rd // 2]
    n[..., : rd // 2] = rb(lo * c - hi * s)
    n[..., rd // 2: rd] = rb(lo * s + hi * c)
    return n


def test_hd256_prep_gate_and_decode_prep(lib):
    nq, nkv, hd, rd, T, start, max_seq = 16, 4, 256, 64, 5, 3, 32
    cosb, sinb = O.precompute_rope(rd, 4096, 1e7)
    cos, sin = f32(cosb).reshape(4096, rd), f32(sinb).reshape(4096, rd)
    qf, k, v = rnd((T, nq, 2, hd), 20, 2.0), rnd((T, nkv, hd), 21, 2.0), rnd((T, nkv, hd), 22)
    qw, kw = rnd((hd,), 23, 0.2), rnd((hd,), 24, 0.2)
    dev = lambda t: t.cuda().contiguous()
    cos_d, sin_d = torch.from_numpy(cosb.view(np.int16)).view(torch.bfloat16).cuda(), torch.from_numpy(sinb.view(np.int16)).view(torch.bfloat16).cuda()
    q_out = torch.zeros((T, nq, hd), dtype=torch.bfloat16, device="cuda")
    kc = torch.zeros((nkv, max_seq, hd), dtype=torch.bfloat16, device="cuda")
    vc = torch.zeros_like(kc)
    sp = torch.tensor([start], dtype=torch.int32, device="cuda")
    qf_d, k_d, v_d, qw_d, kw_d = dev(qf), dev(k), dev(v), dev(qw), dev(kw)
    lib.prefill_attention_hd256_prep_cuda(qf_d.data_ptr(), k_d.data_ptr(), v_d.data_ptr(), qw_d.data_ptr(), kw_d.data_ptr(), cos_d.data_ptr(),
                                          sin_d.data_ptr(), q_out.data_ptr(), kc.data_ptr(), vc.data_ptr(), nq, nkv, T, sp.data_ptr(), rd, 1e-6,
                                          max_seq, st())
    torch.cuda.synchronize()
    for t in range(T):
        wq = _norm_rope_ref(vals(qf[t, :, 0]), vals(qw), cos, sin, start + t, rd, 1e-6)
        wk = _norm_rope_ref(vals(k[t]), vals(kw), cos, sin, start + t, rd, 1e-6)
        assert_bf16_close(bits(q_out[t]), O.f32_to_bf16(wq), 2, floor=2 ** -6, what="q prep")
        assert_bf16_close(bits(kc[:, start + t]), O.f32_to_bf16(wk), 2, floor=2 ** -6, what="k prep")
        assert (bits(vc[:, start + t]) == bits(v[t])).all()
    # gate
    attn = rnd((T, nq, hd), 25)
    attn_d = dev(attn)
    lib.attention_gate_batch_hd256_cuda(qf_d.data_ptr(), attn_d.data_ptr(), nq, T, st())
    want = O.f32_to_bf16(vals(attn) * (1.0 / (1.0 + np.exp(-vals(qf[:, :, 1]), dtype=np.float32))))
    assert_bf16_close(bits(attn_d), want, 1, what="gate")
    # batched decode prep: per-request positions, K in place
    pos = np.array([7, 0, 100, 4095, 33], np.int32)
    k2 = dev(k)
    q2 = torch.zeros((T, nq, hd), dtype=torch.bfloat16, device="cuda")
    pos_d = torch.tensor(pos, device="cuda")
    lib.qk_norm_partial_rope_batched_decode_hd256_cuda(qf_d.data_ptr(), k2.data_ptr(), qw_d.data_ptr(), kw_d.data_ptr(), cos_d.data_ptr(),
                                                       sin_d.data_ptr(), pos_d.data_ptr(), q2.data_ptr(), nq, nkv, T, rd, 1e-6, st())
    torch.cuda.synchronize()
    for t in range(T):
        assert_bf16_close(bits(q2[t]), O.f32_to_bf16(_norm_rope_ref(vals(qf[t, :, 0]), vals(qw), cos, sin, int(pos[t]), rd, 1e-6)), 2,
                          floor=2 ** -6, what="q decode prep")
        assert_bf16_close(bits(k2[t]), O.f32_to_bf16(_norm_rope_ref(vals(k[t]), vals(kw), cos, sin, int(pos[t]), rd, 1e-6)), 2,
                          floor=2 ** -6, what="k decode prep")


@pytest.mark.parametrize("seq_lens", [[1], [100], [700, 33]])
def test_paged_attention_decode_hd256(lib, seq_lens):
    nq, nkv, hd, bs, L = 16, 4, 256, len(seq_lens), 2
    rng = np.random.RandomState(7)
    need = [-(-s // 16) for s in seq_lens]
    ids = rng.permutation(np.arange(1, sum(need) + 3))
    pi, ip, lpl, off = [], [0], [], 0
    for s, n in zip(seq_lens, need):
        pi += ids[off:off + n].tolist(); off += n
        ip.append(len(pi)); lpl.append(((s - 1) % 16) + 1)
    block = 16 * nkv * hd                    # one K (or V) block of a page
    layer_stride, page_stride = 2 * block, L * 2 * block
    layer = 1
    k_off, v_off = layer * layer_stride, layer * layer_stride + block
    kv = rnd(((sum(need) + 4) * page_stride,), 30)
    q = rnd((bs, nq, hd), 31)
    kv_d, q_d = kv.cuda(), q.cuda()
    out = torch.zeros((bs, nq, hd), dtype=torch.bfloat16, device="cuda")
    dv = lambda a: torch.tensor(np.asarray(a, np.int32), device="cuda")
    pi_d, ip_d, lpl_d, req_d, z_d = dv(pi), dv(ip), dv(lpl), dv(np.arange(bs)), dv(np.zeros(bs))
    sm = 1 / math.sqrt(hd)
    rc = lib.paged_attention_decode_cuda_hd256(q_d.data_ptr(), out.data_ptr(), kv_d.data_ptr(), k_off, v_off, pi_d.data_ptr(), ip_d.data_ptr(),
                                               lpl_d.data_ptr(), req_d.data_ptr(), z_d.data_ptr(), z_d.data_ptr(), nq, nkv, hd, 16, bs,
                                               page_stride, sm, st())
    assert rc == 0
    torch.cuda.synchronize()
    kvv, qv = vals(kv), vals(q)
    want = np.zeros((bs, nq, hd), np.float32)
    for b, s in enumerate(seq_lens):
        pages = pi[ip[b]:ip[b + 1]]
        K = np.stack([kvv[pages[t // 16] * page_stride + k_off + (t % 16) * nkv * hd:][:nkv * hd].reshape(nkv, hd) for t in range(s)])
        V = np.stack([kvv[pages[t // 16] * page_stride + v_off + (t % 16) * nkv * hd:][:nkv * hd].reshape(nkv, hd) for t in range(s)])
        for h in range(nq):
            sc = (K[:, h // 4] @ qv[b, h]).astype(np.float32) * np.float32(sm)
            p = np.exp(sc - sc.max(), dtype=np.float32)
            want[b, h] = (p @ V[:, h // 4]) / p.sum(dtype=np.float32)
    assert_bf16_close(bits(out), O.f32_to_bf16(want), 3, floor=float(np.abs(want).max()) / 32, what="hd256 decode attention")


@pytest.mark.parametrize("starts,lens", [([0], [128]), ([0], [77]), ([0, 0, 0], [33, 100, 5]), ([40, 0], [50, 300]), ([0], [1024])])
def test_batch_prefill_paged_hd256(lib, starts, lens):
    """HD-256 causal GQA prefill attention over the paged pool vs the oracle's FA2 restatement (P rounded to bf16,
    denominator of the rounded P), incl. chunked prefill (a request that already holds `start` tokens)."""
    nq, nkv, hd, L, layer = 16, 4, 256, 2, 1
    bs = len(lens)
    kv_lens = [a + b for a, b in zip(starts, lens)]
    rng = np.random.RandomState(11)
    need = [-(-s // 16) for s in kv_lens]
    ids = rng.permutation(np.arange(1, sum(need) + 3))
    pi, ip, lpl, off = [], [0], [], 0
    for s_, n in zip(kv_lens, need):
        pi += ids[off:off + n].tolist(); off += n
        ip.append(len(pi)); lpl.append(((s_ - 1) % 16) + 1)
    block = 16 * nkv * hd
    layer_stride, page_stride = 2 * block, L * 2 * block
    k_off, v_off = layer * layer_stride, layer * layer_stride + block
    kv = rnd(((sum(need) + 4) * page_stride,), 40)
    T = sum(lens)
    q = rnd((T, nq * hd), 41)
    qi = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    dv = lambda a: torch.tensor(np.asarray(a, np.int32), device="cuda")
    kv_d, q_d = kv.cuda(), q.cuda()
    out = torch.zeros((T, nq * hd), dtype=torch.bfloat16, device="cuda")
    pi_d, ip_d, lpl_d, qi_d, z_d = dv(pi), dv(ip), dv(lpl), dv(qi), dv(np.zeros(4096))
    tn = torch.tensor([T], dtype=torch.int32, device="cuda")
    sm = 1 / math.sqrt(hd)
    rc = lib.batch_prefill_paged_cuda_hd256(q_d.data_ptr(), out.data_ptr(), kv_d.data_ptr(), k_off, v_off, pi_d.data_ptr(), ip_d.data_ptr(),
                                            lpl_d.data_ptr(), qi_d.data_ptr(), z_d.data_ptr(), z_d.data_ptr(), z_d.data_ptr(), z_d.data_ptr(),
                                            tn.data_ptr(), nq, nkv, hd, 16, T, bs, 1, page_stride, sm, st())
    assert rc == 0
    torch.cuda.synchronize()
    want = O.batch_prefill_paged(bits(q), bits(kv), k_off, v_off, np.array(pi, np.int32), np.array(ip, np.int32), np.array(lpl, np.int32),
                                 qi, nq, nkv, hd, 16, page_stride, sm)
    # FA2 rounds P against the RUNNING row max, the oracle against the final one (qwen3_oracle.c a8 note): with 256-long
    # dot products and up to 1024 keys a few outputs land 4 ulp apart (measured worst 4.0 on B200)
    assert_bf16_close(bits(out), want, 5, floor=float(np.abs(f32(want)).max()) / 32, what="hd256 prefill attention")


def test_hybrid_model_bringup_matches_oracle(lib):
    """End to end through the C ABI (tests/tools/qwen35_bringup.py): 24 teacher-forced steps of a tiny hybrid model."""
    import importlib.util
    p = os.path.join(os.path.dirname(__file__), "tools", "qwen35_bringup.py")
    spec = importlib.util.spec_from_file_location("qwen35_bringup", p)
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    assert mod.run()


def test_gated_delta_rule_prefill_recurrent(lib):
    nk, nv, dk, dv, T = 16, 32, 128, 128, 37
    g = torch.Generator().manual_seed(14)
    qkv = rnd((T, 2 * nk * dk + nv * dv), 15)
    a, b, dtb = rnd((T, nv), 16), rnd((T, nv), 17), rnd((nv,), 18, 0.5)
    a_log = torch.randn(nv, generator=g) * 0.5
    S = (torch.randn((nv, dk, dv), generator=g) * 0.1).float()
    qkv_d, a_d, b_d, dtb_d, alog_d, Sd = qkv.cuda(), a.cuda(), b.cuda(), dtb.cuda(), a_log.cuda(), S.cuda()
    out = torch.empty((T, nv * dv), dtype=torch.bfloat16, device="cuda")
    rc = lib.pk_b200_gated_delta_rule_prefill_recurrent(qkv_d.data_ptr(), b_d.data_ptr(), a_d.data_ptr(), dtb_d.data_ptr(), alog_d.data_ptr(),
                                                        Sd.data_ptr(), out.data_ptr(), nk, nv, dk, dv, T, st())
    assert rc == 0
    torch.cuda.synchronize()
    qv, av, bv = vals(qkv), vals(a), vals(b)
    Sw = S.numpy().copy()
    want = np.stack([gated_delta_rule_step(qv[t, :nk * dk].reshape(nk, dk), qv[t, nk * dk:2 * nk * dk].reshape(nk, dk),
                                           qv[t, 2 * nk * dk:].reshape(nv, dv), av[t], bv[t], vals(dtb), a_log.numpy(), Sw).reshape(-1)
                     for t in range(T)])
    assert_bf16_close(bits(out), O.f32_to_bf16(want), 2, floor=float(np.abs(want).max()) / 64, what="gdr sequence out")
    np.testing.assert_allclose(Sd.cpu().numpy(), Sw, rtol=2e-4, atol=2e-5)


@pytest.mark.parametrize("N", [1, 2])
def test_gemv_qwen35_prologue_and_rounded_swiglu(lib, N):
    """pk_b200_gemv_fused x_mode 3 (hidden_out = bf16(X + residual), x = (1 + w) RMSNorm of that ROUNDED sum,
    ops/norm.rs rms_norm_offset after ops/elementwise.rs add) with the linear-attention segment split (qkv | z | [b; a]),
    and epi 4 (act = bf16(bf16(silu(gate)) * up): Qwen3.5 keeps the unfused silu_mul's two roundings)."""
    import ctypes as C
    H, qkvd, zd, nv, inter = 2560, 8192, 4096, 32, 9216
    hid, res, nw = rnd((N, H), 70, 1.0), rnd((N, H), 71, 0.3), rnd((H,), 72, 0.2)
    W = rnd((qkvd + zd + 2 * nv, H), 73, 0.02)
    outs = [torch.zeros((N, n), dtype=torch.bfloat16, device="cuda") for n in (qkvd, zd, 2 * nv)]
    hout = torch.zeros((N, H), dtype=torch.bfloat16, device="cuda")
    keep = [hid.cuda(), res.cuda(), nw.cuda(), W.cuda()]
    g = ffi.GemvArgs()
    g.W, g.X = keep[3].data_ptr(), keep[0].data_ptr()
    g.Y = (C.c_void_p * 3)(*[o.data_ptr() for o in outs])
    g.seg_rows = (C.c_int * 3)(qkvd, zd, 2 * nv)
    g.M, g.N, g.K, g.x_mode, g.epi = qkvd + zd + 2 * nv, N, H, 3, 0
    g.residual, g.norm_w, g.eps, g.hidden_out, g.normed_out = keep[1].data_ptr(), keep[2].data_ptr(), 1e-6, hout.data_ptr(), None
    assert lib.pk_b200_gemv_fused(C.byref(g), st()) == 0
    torch.cuda.synchronize()
    summed = rb(vals(hid) + vals(res))
    assert (bits(hout) == O.f32_to_bf16(summed)).all()
    want = O.f32_to_bf16(rms_norm_offset(summed, vals(nw), 1e-6) @ vals(W).T)
    got = np.concatenate([bits(o) for o in outs], axis=1)
    assert_bf16_close(got, want, 2, floor=float(np.abs(f32(want)).max()) / 64, frac_exact=0.85, what="x_mode 3 in-projection")
    # epi 4 on a gate | up matrix
    Wgu, x = rnd((2 * inter, H), 74, 0.02), rnd((N, H), 75, 1.0)
    act = torch.zeros((N, inter), dtype=torch.bfloat16, device="cuda")
    keep2 = [Wgu.cuda(), x.cuda(), torch.zeros((N, H), dtype=torch.bfloat16, device="cuda")]
    g2 = ffi.GemvArgs()
    g2.W, g2.X = keep2[0].data_ptr(), keep2[1].data_ptr()
    g2.Y = (C.c_void_p * 3)(act.data_ptr(), None, None)
    g2.seg_rows = (C.c_int * 3)(inter, 0, 0)
    g2.M, g2.N, g2.K, g2.x_mode, g2.epi = inter, N, H, 0, 4
    assert lib.pk_b200_gemv_fused(C.byref(g2), st()) == 0
    torch.cuda.synchronize()
    gu = rb(vals(x) @ vals(Wgu).T)
    want = O.f32_to_bf16(rb(silu(gu[:, :inter])) * gu[:, inter:])
    assert_bf16_close(bits(act), want, 2, floor=float(np.abs(f32(want)).max()) / 64, frac_exact=0.85, what="epi 4 rounded swiglu")
