"""What a user of this framework has it do, as cases that can be timed and compared: whole requests of the served Qwen3 model and the blocks
that its decoders are made of, each through the entry points that a program calls (``Qwen3Model`` and the C ABI behind ``ffi``).

A case is a dict of plain values.  ``prepare`` makes what a program has in hand before the call (weights, caches, plans, inputs; from the seed
alone), ``run`` is one pass, ``exact`` the same pass in plain 64-bit torch, ``work`` the bytes and operations that a pass cannot do without.
"""
import ctypes as C
import math
import random

import torch

from pegainfer_b200 import ffi
from pegainfer_b200.config import PRESETS
from pegainfer_b200.model import ModelRuntimeConfig, Qwen3Model
from pegainfer_b200.qwen35 import QWEN35_4B

BF16, F32, F64, I32 = torch.bfloat16, torch.float32, torch.float64, torch.int32
PAGE = 16            # slots of a cache page
POSITIONS = 4096     # rotary table and longest context of the Qwen3 path
EPS = 1e-6
GROUPED_FROM = 32    # tokens from which the experts run bucketed (as the layer-list host does)


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # a short chat turn of one user: 128-token prompt, then decoded tokens one by one (CUDA graph, batch 1)
        dict(name="chat", kind="model", model="qwen3-4b", prompt=128, decode=16),
        # time to the first token of a long prompt
        dict(name="prompt", kind="model", model="qwen3-4b", prompt=2048, decode=0),
        # feed-forward of one decoded token, of a batch of decoding requests, and of a long prompt portion of odd length
        dict(name="mlp_1", kind="mlp", model="qwen3-4b", tokens=1),
        dict(name="mlp_48", kind="mlp", model="qwen3-8b", tokens=48),
        dict(name="mlp_3001", kind="mlp", model="qwen3-8b", tokens=3001),
        # attention block of a decoding batch (contexts of different lengths) and of three prompts batched together
        dict(name="attn_decode", kind="attention", model="qwen3-4b", requests=24, tokens=24, cached=2600),
        dict(name="attn_prompts", kind="attention", model="qwen3-4b", requests=3, tokens=3333, cached=0),
        # linear-attention layer of the hybrid model over a 1024-token prompt
        dict(name="hybrid", kind="hybrid", tokens=1024, carried=False),
        # routed experts of a prompt
        dict(name="experts", kind="experts", tokens=2048, width=2048, ff=1408, experts=64, top=6, act=1),
        # grouped-query attention of the layer-list designs, decode step of four requests: the smallest call
        dict(name="gqa_step", kind="gqa", requests=4, tokens=4, cached=2048, heads=16, kv_heads=4, dim=128, window=1024, softcap=0.0, gated=False, f32=False),
        # attention over the compressed cache, whole prompt
        dict(name="latent", kind="latent", requests=1, tokens=2048, cached=0, heads=16, rank=512, rot=64, window=0),
        # gated delta rule of the layer-list designs over a prompt
        dict(name="delta", kind="delta", requests=1, tokens=2048, heads=16, kv_heads=8, dim=128, f32=False),
    ]


def _log(rng, lo, hi):
    """a whole number between lo and hi, spread over its logarithm"""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["model", "mlp", "mlp", "attention", "attention", "hybrid", "experts", "gqa", "latent", "delta"])
    model = rng.choice(["qwen3-4b", "qwen3-8b"])
    if kind == "model":
        return dict(kind=kind, model="qwen3-4b", prompt=_log(rng, 16, 2048), decode=rng.randint(0, 16))
    if kind == "mlp":
        return dict(kind=kind, model=model, tokens=_log(rng, 1, 4096))
    if kind == "attention":
        if rng.random() < 0.5:  # decode step
            n = _log(rng, 1, 64)
            return dict(kind=kind, model=model, requests=n, tokens=n, cached=_log(rng, 16, 3000))
        n = rng.randint(1, 6)
        return dict(kind=kind, model=model, requests=n, tokens=_log(rng, 8 * n, 3500), cached=rng.choice([0, 0, rng.randint(1, 500)]))
    if kind == "hybrid":
        return dict(kind=kind, tokens=_log(rng, 16, 2048), carried=rng.random() < 0.3)
    if kind == "experts":
        width, ff, experts, top = rng.choice([(2048, 1408, 64, 6), (1024, 768, 16, 2)])
        return dict(kind=kind, tokens=_log(rng, 1, 2048), width=width, ff=ff, experts=experts, top=top, act=rng.randint(0, 1))
    heads = rng.choice([8, 16])
    step = rng.random() < 0.5
    n = rng.randint(1, 6)
    tokens = n if step else _log(rng, 8 * n, 2048)
    if kind == "gqa":
        f32 = rng.random() < 0.2
        return dict(kind=kind, requests=n, tokens=min(tokens, 300) if f32 else tokens, cached=_log(rng, 16, 2500) if step else rng.choice([0, rng.randint(1, 500)]),
                    heads=heads, kv_heads=heads // rng.choice([2, 4]), dim=rng.choice([64, 128]), window=rng.choice([0, 1024]),
                    softcap=rng.choice([0.0, 30.0]), gated=rng.random() < 0.5, f32=f32)
    if kind == "latent":
        rank, rot = rng.choice([(512, 64), (256, 32)])
        return dict(kind=kind, requests=n, tokens=tokens, cached=_log(rng, 16, 2500) if step else 0, heads=heads, rank=rank, rot=rot, window=rng.choice([0, 1024]))
    return dict(kind="delta", requests=n, tokens=tokens, heads=heads, kv_heads=heads // rng.choice([1, 2]), dim=rng.choice([64, 128]), f32=rng.random() < 0.2)


def _share(total, parts, key):
    """`total` cut into `parts` unequal whole parts, each at least one"""
    r = random.Random("%s %d %d" % (key, total, parts))
    w = [r.uniform(0.4, 1.6) for _ in range(parts)]
    cut = [1 + int((total - parts) * x / sum(w)) for x in w]
    cut[-1] += total - sum(cut)
    return cut


def _rows(case):
    """(new tokens, tokens already cached) of every request"""
    n, t, c = case["requests"], case["tokens"], case["cached"]
    lens = _share(t, n, "tokens") if t > n else [1] * n
    if c == 0:
        had = [0] * n
    elif t > n:
        had = [c] * n
    else:  # decode step: contexts between a quarter of `cached` and all of it
        r = random.Random("cached %d %d" % (n, c))
        had = [c if i == 0 else r.randint(max(1, c // 4), c) for i in range(n)]
    return lens, had


# ------------------------------------------------------------------ small helpers
_ready = []


def _lib():
    lib = ffi.lib()
    if not _ready:  # once per thread that launches, as the hosts do
        lib.cuda_set_device(0)
        lib.cublas_init()
        lib.pk_b200_set_pdl(1)
        _ready.append(True)
    return lib


def _ok(rc):
    if rc != 0:
        raise RuntimeError("a kernel entry returned %d" % rc)


def _stream():
    return torch.cuda.current_stream().cuda_stream


class _Maker:
    """tensors of one seed on the GPU"""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(seed)

    def normal(self, shape, std=1.0, dtype=BF16, mean=0.0):
        return torch.empty(shape, dtype=dtype, device="cuda").normal_(mean, std, generator=self.g)

    def shuffled(self, n):
        return torch.randperm(n, generator=self.g, device="cuda").tolist()


def _ints(v):
    return torch.tensor(v, dtype=I32, device="cuda")


def _pages(mk, lens):
    """scrambled pages for contexts of these lengths: (pages per request, number of pages)"""
    need = [(n + PAGE - 1) // PAGE for n in lens]
    order = [p + 1 for p in mk.shuffled(sum(need) + 2)]  # page 0 stays free, as in the framework's pool
    out, at = [], 0
    for n in need:
        out.append(order[at:at + n])
        at += n
    return out, sum(need) + 3


def _rope_tables(dim, base=1e6):
    inv = base ** (-torch.arange(0, dim, 2, dtype=F32, device="cuda") / dim)
    ang = torch.arange(POSITIONS, dtype=F32, device="cuda")[:, None] * inv
    return torch.cat([ang.cos()] * 2, 1).to(BF16).contiguous(), torch.cat([ang.sin()] * 2, 1).to(BF16).contiguous()


def _rms(x, w, eps=EPS):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * w


def _silu(x):
    return x * torch.sigmoid(x)


def _rope_half(x, cos, sin):
    """x [tokens, heads, dim], cos / sin [tokens, dim]: pairs (i, i + dim / 2)"""
    a, b = x.chunk(2, -1)
    return x * cos[:, None] + torch.cat([-b, a], -1) * sin[:, None]


def _causal(q, k, v, scale, first):
    """softmax attention in 64 bits: q [n, H, D] at positions first.., k / v [m, G, D]"""
    n, H, _ = q.shape
    m, G, _ = k.shape
    at = torch.arange(m, device=q.device)
    hidden = at[None, :] > (torch.arange(n, device=q.device) + first)[:, None]
    out = torch.empty(n, H, v.shape[-1], dtype=q.dtype, device=q.device)
    for h in range(H):
        s = (q[:, h] @ k[:, h * G // H].T) * scale
        out[:, h] = torch.softmax(s.masked_fill(hidden, -math.inf), -1) @ v[:, h * G // H]
    return out


# ------------------------------------------------------------------ whole model
def _model_weights(cfg, seed):
    """random checkpoint of the model's shape under its tensor names: a residual stream of unit size that every layer adds a little to, as in a
    trained model (what a layer writes is scaled by the depth), norms near one"""
    mk = _Maker(seed)
    c = cfg
    write = 0.02 / math.sqrt(2 * c.num_hidden_layers)
    yield "model.embed_tokens.weight", mk.normal((c.vocab_size, c.hidden_size), 1.0)
    for i in range(c.num_hidden_layers):
        p = "model.layers.%d." % i
        yield p + "input_layernorm.weight", mk.normal((c.hidden_size,), 0.1, mean=1.0)
        yield p + "self_attn.q_proj.weight", mk.normal((c.q_dim, c.hidden_size), 0.02)
        yield p + "self_attn.k_proj.weight", mk.normal((c.kv_dim, c.hidden_size), 0.02)
        yield p + "self_attn.v_proj.weight", mk.normal((c.kv_dim, c.hidden_size), 0.02)
        yield p + "self_attn.o_proj.weight", mk.normal((c.hidden_size, c.q_dim), write)
        yield p + "self_attn.q_norm.weight", mk.normal((c.head_dim,), 0.1, mean=1.0)
        yield p + "self_attn.k_norm.weight", mk.normal((c.head_dim,), 0.1, mean=1.0)
        yield p + "post_attention_layernorm.weight", mk.normal((c.hidden_size,), 0.1, mean=1.0)
        yield p + "mlp.gate_proj.weight", mk.normal((c.intermediate_size, c.hidden_size), 0.02)
        yield p + "mlp.up_proj.weight", mk.normal((c.intermediate_size, c.hidden_size), 0.02)
        yield p + "mlp.down_proj.weight", mk.normal((c.hidden_size, c.intermediate_size), write)
    yield "model.norm.weight", mk.normal((c.hidden_size,), 0.1, mean=1.0)
    if not c.tie_word_embeddings:
        yield "lm_head.weight", mk.normal((c.vocab_size, c.hidden_size), 0.02)


def _model_tokens(case, seed):
    r = random.Random(seed)
    vocab = PRESETS[case["model"]].vocab_size
    return [r.randrange(100, vocab) for _ in range(case["prompt"])], [r.randrange(100, vocab) for _ in range(case["decode"])]


def _prepare_model(case, seed):
    cfg = PRESETS[case["model"]]
    pages = (case["prompt"] + case["decode"]) // PAGE + 8
    m = Qwen3Model(cfg, _model_weights(cfg, seed), ModelRuntimeConfig(num_pages=pages, max_batch=1))
    prompt, forced = _model_tokens(case, seed)
    return dict(model=m, prompt=prompt, forced=forced)


def _run_model(case, s):
    m = s["model"]
    kv = m.alloc_kv()
    out = [m.prefill([s["prompt"]], [kv])]
    out += [m.decode([t], [kv])[0] for t in s["forced"]]
    m.drop_request(kv)
    return torch.cat(out)


def _exact_model(case, seed):
    cfg = PRESETS[case["model"]]
    prompt, forced = _model_tokens(case, seed)
    ids = torch.tensor(prompt + forced, device="cuda")
    T, c = len(ids), cfg
    cos, sin = (t[:T].to(F64) for t in _rope_tables(c.head_dim, c.rope_theta))
    x, w, layer, embed = None, {}, "", None
    for name, t in _model_weights(cfg, seed):
        if name == "model.embed_tokens.weight":
            embed = t
            x = embed[ids].to(F64)
            continue
        if name in ("model.norm.weight", "lm_head.weight"):
            w[name] = t
            continue
        _, _, layer, leaf = name.split(".", 3)
        w[leaf] = t.to(F64)
        if leaf != "mlp.down_proj.weight":
            continue
        h = _rms(x, w["input_layernorm.weight"], c.rms_norm_eps)
        q = _rms((h @ w["self_attn.q_proj.weight"].T).view(T, -1, c.head_dim), w["self_attn.q_norm.weight"], c.rms_norm_eps)
        k = _rms((h @ w["self_attn.k_proj.weight"].T).view(T, -1, c.head_dim), w["self_attn.k_norm.weight"], c.rms_norm_eps)
        v = (h @ w["self_attn.v_proj.weight"].T).view(T, -1, c.head_dim)
        a = _causal(_rope_half(q, cos, sin), _rope_half(k, cos, sin), v, c.head_dim ** -0.5, 0)
        x = x + a.reshape(T, -1) @ w["self_attn.o_proj.weight"].T
        h = _rms(x, w["post_attention_layernorm.weight"], c.rms_norm_eps)
        x = x + (_silu(h @ w["mlp.gate_proj.weight"].T) * (h @ w["mlp.up_proj.weight"].T)) @ w["mlp.down_proj.weight"].T
        w = {}
    head = w.get("lm_head.weight", embed)
    x = _rms(x[case["prompt"] - 1:], w["model.norm.weight"].to(F64), c.rms_norm_eps)
    return torch.cat([x @ head[r:r + 16384].to(F64).T for r in range(0, c.vocab_size, 16384)], 1)


def _work_model(case):
    c = PRESETS[case["model"]]
    P, D, L = case["prompt"], case["decode"], c.num_hidden_layers
    layer = c.hidden_size * (2 * c.q_dim + 2 * c.kv_dim) + 3 * c.hidden_size * c.intermediate_size
    head = c.vocab_size * c.hidden_size
    pairs = P * (P + 1) // 2 + sum(P + i + 1 for i in range(D))
    kv = sum(P + i + 1 for i in range(D)) * 2 * c.kv_dim * L * 2
    return {"bytes": 2 * (1 + D) * (layer * L + head) + kv + (1 + D) * c.vocab_size * 2,
            "flops": 2 * (P + D) * layer * L + 2 * (1 + D) * head + 4 * pairs * c.q_dim * L}


# ------------------------------------------------------------------ feed-forward block
def _prepare_mlp(case, seed):
    cfg, T, mk = PRESETS[case["model"]], case["tokens"], _Maker(seed)
    H, I = cfg.hidden_size, cfg.intermediate_size
    new = lambda *shape: torch.empty(shape, dtype=BF16, device="cuda")  # noqa: E731
    return dict(lib=_lib(), T=T, H=H, I=I, hidden=mk.normal((T, H)), residual=mk.normal((T, H), 0.5), norm=mk.normal((H,), 0.1, mean=1.0),
                gate_up=mk.normal((2 * I, H), 0.02), down=mk.normal((H, I), 0.02), hidden_out=new(T, H), normed=new(T, H), gu=new(T, 2 * I) if T > 4 else None,
                act=new(T, I), y=new(T, H), out=new(T, H))


def _gemv(lib, st, W, X, Y, M, N, K, **more):
    g = ffi.GemvArgs()
    g.W, g.X, g.M, g.N, g.K = W.data_ptr(), X.data_ptr(), M, N, K
    ys = Y if isinstance(Y, tuple) else (Y,)
    rows = more.pop("rows", (M,))
    for i, y in enumerate(ys):
        g.Y[i], g.seg_rows[i] = y.data_ptr(), rows[i]
    for k, v in more.items():
        setattr(g, k, v.data_ptr() if isinstance(v, torch.Tensor) else v)
    _ok(lib.pk_b200_gemv_fused(C.byref(g), st))


def _run_mlp(case, s):
    lib, T, H, I, st = s["lib"], s["T"], s["H"], s["I"], _stream()
    p = {k: v.data_ptr() for k, v in s.items() if isinstance(v, torch.Tensor)}
    if T <= 4:  # decode: sum and norm in the first product's prologue, activation in its epilogue
        _gemv(lib, st, s["gate_up"], s["hidden"], s["act"], I, T, H, x_mode=1, residual=s["residual"], norm_w=s["norm"], eps=EPS,
              hidden_out=s["hidden_out"], epi=1)
        _gemv(lib, st, s["down"], s["act"], s["y"], H, T, I)
        return {"hidden": s["hidden_out"], "out": s["y"]}
    lib.rms_norm_batched_cuda(p["hidden"], p["norm"], p["normed"], H, T, EPS, st)
    if lib.pk_b200_gemm_swiglu(p["gate_up"], p["normed"], p["act"], I, T, H, st) != 0:  # not a shape for the one-launch form
        lib.gemm_cuda(p["gate_up"], p["normed"], p["gu"], 2 * I, T, H, st)
        lib.silu_mul_fused_cuda(p["gu"], p["act"], I, T, st)
    lib.gemm_cuda(p["down"], p["act"], p["y"], H, T, I, st)
    _ok(lib.add_cuda(p["hidden"], p["y"], p["out"], H * T, st))
    return {"out": s["out"]}


def _exact_mlp(case, seed):
    s = _prepare_mlp(case, seed)
    d = {k: v.to(F64) for k, v in s.items() if k in ("hidden", "residual", "norm", "gate_up", "down")}
    few = case["tokens"] <= 4
    x = d["hidden"] + d["residual"] if few else d["hidden"]
    gu = _rms(x, d["norm"]) @ d["gate_up"].T
    y = (_silu(gu[:, :s["I"]]) * gu[:, s["I"]:]) @ d["down"].T
    return {"hidden": x, "out": y} if few else {"out": d["hidden"] + y}


def _work_mlp(case):
    c, T = PRESETS[case["model"]], case["tokens"]
    w = 3 * c.hidden_size * c.intermediate_size
    return {"bytes": 2 * w + 2 * T * c.hidden_size * (4 if T <= 4 else 2), "flops": 2 * T * w}


# ------------------------------------------------------------------ attention block of the Qwen3 path
def _prepare_attention(case, seed):
    cfg, mk, lib = PRESETS[case["model"]], _Maker(seed), _lib()
    H, qd, kd, hd, nkv = cfg.hidden_size, cfg.q_dim, cfg.kv_dim, cfg.head_dim, cfg.num_key_value_heads
    lens, had = _rows(case)
    T, n = sum(lens), len(lens)
    kv_len = [a + b for a, b in zip(lens, had)]
    pages, n_pages = _pages(mk, kv_len)
    pool = torch.zeros((n_pages, 2, PAGE, nkv, hd), dtype=BF16, device="cuda")
    for pg, h in zip(pages, had):
        if h:
            full = torch.zeros(2, len(pg) * PAGE, nkv, hd, dtype=BF16, device="cuda")
            full[:, :h] = mk.normal((2, h, nkv, hd))
            pool[torch.tensor(pg, device="cuda")] = full.view(2, len(pg), PAGE, nkv, hd).transpose(0, 1)
    cos, sin = _rope_tables(hd, cfg.rope_theta)
    decode = T == n
    new = lambda *shape: torch.empty(shape, dtype=BF16, device="cuda")  # noqa: E731
    s = dict(lib=lib, cfg=cfg, lens=lens, had=had, T=T, decode=decode, pages=pages, pool=pool, cos=cos, sin=sin,
             hidden=mk.normal((T, H)), residual=mk.normal((T, H), 0.5), norm=mk.normal((H,), 0.1, mean=1.0), qkv=mk.normal((qd + 2 * kd, H), 0.02),
             o=mk.normal((H, qd), 0.02), qn=mk.normal((hd,), 0.1, mean=1.0), kn=mk.normal((hd,), 0.1, mean=1.0), hidden_out=new(T, H), normed=new(T, H),
             q=new(T, qd), k=new(T, kd), v=new(T, kd), att=new(T, qd), out=new(T, H))
    ptr = [0]
    for pg in pages:
        ptr.append(ptr[-1] + len(pg))
    s.update(indices=_ints([x for pg in pages for x in pg]), indptr=_ints(ptr), last=_ints([(x - 1) % PAGE + 1 for x in kv_len]),
             positions=_ints([h + t for h, m in zip(had, lens) for t in range(m)]), batch=_ints([i for i, m in enumerate(lens) for _ in range(m)]),
             chunk=_ints(kv_len))
    if decode:
        most = POSITIONS // 64 + 1
        s.update(most=most, partial=torch.empty(n * most * cfg.num_attention_heads * (hd + 2), dtype=F32, device="cuda"),
                 counters=torch.zeros(n * nkv, dtype=I32, device="cuda"))
        return s
    tile = lib.batch_prefill_cta_tile_q_with_override(T, cfg.num_attention_heads, nkv, hd, 64)
    group, req, qt, q_ptr = cfg.num_attention_heads // nkv, [], [], [0]
    for i, m in enumerate(lens):
        q_ptr.append(q_ptr[-1] + m)
        for t in range((m * group + tile - 1) // tile):
            req.append(i)
            qt.append(t)
    s.update(tile=tile, tiles=len(req), q_indptr=_ints(q_ptr), request=_ints(req), q_tile=_ints(qt), kv_tile=_ints([0] * len(req)), rows=_ints([T]))
    return s


def _run_attention(case, s):
    lib, c, T, st = s["lib"], s["cfg"], s["T"], _stream()
    p = {k: v.data_ptr() for k, v in s.items() if isinstance(v, torch.Tensor)}
    H, qd, kd, nh, nkv, hd = c.hidden_size, c.q_dim, c.kv_dim, c.num_attention_heads, c.num_key_value_heads, c.head_dim
    v_off, stride, n, scale = PAGE * nkv * hd, 2 * PAGE * nkv * hd, len(s["lens"]), hd ** -0.5
    few = s["decode"] and T <= 4
    if few:
        _gemv(lib, st, s["qkv"], s["hidden"], (s["q"], s["k"], s["v"]), qd + 2 * kd, T, H, rows=(qd, kd, kd), x_mode=1, residual=s["residual"],
              norm_w=s["norm"], eps=EPS, hidden_out=s["hidden_out"])
    else:
        lib.rms_norm_batched_cuda(p["hidden"], p["norm"], p["normed"], H, T, EPS, st)
        _ok(lib.pk_b200_gemm_segments(p["qkv"], p["normed"], (C.c_void_p * 3)(p["q"], p["k"], p["v"]), (C.c_int * 3)(qd, kd, kd), qd + 2 * kd, T, H, st))
    if s["decode"]:
        _ok(lib.pk_b200_decode_attention_fused(p["q"], p["k"], p["v"], p["att"], p["pool"], 0, v_off, p["indices"], p["indptr"], p["last"], p["positions"],
                                               p["qn"], p["kn"], p["cos"], p["sin"], EPS, p["partial"], p["counters"], 64, s["most"], nh, nkv, hd, PAGE, n,
                                               stride, scale, st))
    else:
        if n == 1:
            lib.prefill_qk_norm_rope_only_cuda(p["q"], p["k"], p["qn"], p["kn"], p["cos"], p["sin"], nh, nkv, hd, T, s["had"][0], EPS, st)
        else:
            lib.qk_norm_rope_batched_decode_cuda(p["q"], p["k"], p["qn"], p["kn"], p["cos"], p["sin"], p["positions"], nh, nkv, hd, T, EPS, st)
        _ok(lib.paged_kv_scatter_cuda(p["pool"], 0, v_off, p["indices"], p["indptr"], p["last"], p["k"], p["v"], p["batch"], p["positions"], T, nkv, hd,
                                      PAGE, stride, kd, hd, st))
        _ok(lib.batch_prefill_paged_cuda_with_cta_tile_q(p["q"], p["att"], p["pool"], 0, v_off, p["indices"], p["indptr"], p["last"], p["q_indptr"],
                                                         p["request"], p["q_tile"], p["kv_tile"], p["chunk"], p["rows"], nh, nkv, hd, PAGE, T, n,
                                                         s["tiles"], stride, scale, s["tile"], st))
    if few:
        _gemv(lib, st, s["o"], s["att"], s["out"], H, T, qd)
        return {"hidden": s["hidden_out"], "out": s["out"], "cache": s["pool"]}
    lib.gemm_cuda(p["o"], p["att"], p["out"], H, T, qd, st)
    return {"out": s["out"], "cache": s["pool"]}


def _exact_attention(case, seed):
    s = _prepare_attention(case, seed)
    c, T = s["cfg"], s["T"]
    d = {k: s[k].to(F64) for k in ("hidden", "residual", "norm", "qkv", "o", "qn", "kn", "cos", "sin", "pool")}
    few = s["decode"] and T <= 4
    x = d["hidden"] + d["residual"] if few else d["hidden"]
    qkv = _rms(x, d["norm"]) @ d["qkv"].T
    at = s["positions"].long()
    cos, sin, hd = d["cos"][at], d["sin"][at], c.head_dim
    q = _rope_half(_rms(qkv[:, :c.q_dim].view(T, -1, hd), d["qn"]), cos, sin)
    k = _rope_half(_rms(qkv[:, c.q_dim:c.q_dim + c.kv_dim].view(T, -1, hd), d["kn"]), cos, sin)
    v = qkv[:, c.q_dim + c.kv_dim:].view(T, -1, hd)
    pool, outs, row = d["pool"], [], 0
    for m, h, pg in zip(s["lens"], s["had"], s["pages"]):
        pos = torch.arange(h, h + m, device="cuda")
        page = torch.tensor(pg, device="cuda")
        pool[page[pos // PAGE], 0, pos % PAGE] = k[row:row + m]
        pool[page[pos // PAGE], 1, pos % PAGE] = v[row:row + m]
        kv = pool[page].transpose(0, 1).reshape(2, -1, c.num_key_value_heads, hd)[:, :h + m]
        outs.append(_causal(q[row:row + m], kv[0], kv[1], hd ** -0.5, h))
        row += m
    out = torch.cat(outs).reshape(T, -1) @ d["o"].T
    return {"hidden": x, "out": out, "cache": pool} if few else {"out": out, "cache": pool}


def _work_attention(case):
    c = PRESETS[case["model"]]
    lens, had = _rows(case)
    T, w = sum(lens), 2 * c.hidden_size * (c.q_dim + c.kv_dim)
    pairs = sum(m * h + m * (m + 1) // 2 for m, h in zip(lens, had))
    return {"bytes": 2 * w + 4 * T * c.hidden_size + 4 * c.kv_dim * (sum(had) + T), "flops": 2 * T * w + 4 * pairs * c.q_dim}


# ------------------------------------------------------------------ linear-attention layer of the hybrid model
def _prepare_hybrid(case, seed):
    c, T, mk = QWEN35_4B, case["tokens"], _Maker(seed)
    H, nk, nv, taps = c.hidden_size, c.linear_num_key_heads, c.linear_num_value_heads, c.linear_conv_kernel_dim
    kd, vd = nk * 128, nv * 128
    ch = 2 * kd + vd
    new = lambda *shape: torch.empty(shape, dtype=BF16, device="cuda")  # noqa: E731
    s = dict(lib=_lib(), T=T, H=H, nk=nk, nv=nv, ch=ch, vd=vd, taps=taps, hidden=mk.normal((T, H)), norm=mk.normal((H,), 0.1),
             w_in=mk.normal((ch + vd + 2 * nv, H), 0.5 * H ** -0.5), conv=mk.normal((ch, taps), 0.4), dt_bias=mk.normal((nv,), 0.5),
             a_log=mk.normal((nv,), 0.5, F32), gnorm=mk.normal((128,), 0.2, F32, 1.0), w_out=mk.normal((H, vd), 0.5 * vd ** -0.5),
             state=torch.zeros(nv, 128, 128, dtype=F32, device="cuda"), tail=torch.zeros(ch, taps - 1, dtype=BF16, device="cuda"),
             x=new(T, H), qkv=new(T, ch), z=new(T, vd), b=new(T, nv), a=new(T, nv), mixed=new(T, ch), heads=new(T, vd), gated=new(T, vd), out=new(T, H))
    if case["carried"]:  # a later portion of the prompt: the state that the first one left
        s.update(state0=mk.normal((nv, 128, 128), 0.1, F32), tail0=mk.normal((ch, taps - 1), 0.5))
    return s


def _run_hybrid(case, s):
    lib, T, H, nv, st = s["lib"], s["T"], s["H"], s["nv"], _stream()
    if case["carried"]:
        s["state"].copy_(s["state0"])
        s["tail"].copy_(s["tail0"])
    else:  # a new request starts from nothing
        s["state"].zero_()
        s["tail"].zero_()
    p = {k: v.data_ptr() for k, v in s.items() if isinstance(v, torch.Tensor)}
    ch, vd = s["ch"], s["vd"]
    lib.rms_norm_batched_offset_cuda(p["hidden"], p["norm"], p["x"], H, T, EPS, st)
    _ok(lib.pk_b200_gemm_segments(p["w_in"], p["x"], (C.c_void_p * 3)(p["qkv"], p["z"], p["b"]), (C.c_int * 3)(ch, vd, nv), ch + vd + nv, T, H, st))
    lib.gemm_cuda(p["w_in"] + (ch + vd + nv) * H * 2, p["x"], p["a"], nv, T, H, st)
    lib.conv1d_prefill_cuda(p["qkv"], p["conv"], p["tail"], p["mixed"], ch, T, s["taps"], st)
    _ok(lib.pk_b200_gated_delta_rule_prefill_recurrent(p["mixed"], p["b"], p["a"], p["dt_bias"], p["a_log"], p["state"], p["heads"], s["nk"], nv, 128, 128,
                                                       T, st))
    lib.rms_norm_gated_cuda(p["heads"], p["gnorm"], p["z"], p["gated"], nv * T, 128, EPS, st)
    lib.gemm_cuda(p["w_out"], p["gated"], p["out"], H, T, vd, st)
    return {"out": s["out"], "state": s["state"], "tail": s["tail"]}


def _delta_rule(q, k, v, decay, beta, S):
    """q / k [T, H, D], v [T, H, V], decay / beta [T, H], S [H, D, V] in 64 bits"""
    out = []
    for t in range(q.shape[0]):
        S = S * decay[t][:, None, None]
        u = (v[t] - torch.bmm(k[t][:, None], S)[:, 0]) * beta[t][:, None]
        S = torch.baddbmm(S, k[t][:, :, None], u[:, None])
        out.append(torch.bmm(q[t][:, None], S)[:, 0])
    return torch.stack(out), S


def _exact_hybrid(case, seed):
    s = _prepare_hybrid(case, seed)
    T, H, nk, nv, ch, vd = s["T"], s["H"], s["nk"], s["nv"], s["ch"], s["vd"]
    d = {k: v.to(F64) for k, v in s.items() if isinstance(v, torch.Tensor)}
    z = _rms(d["hidden"], 1 + d["norm"]) @ d["w_in"].T
    qkv, gate, b, a = z[:, :ch], z[:, ch:ch + vd], z[:, ch + vd:ch + vd + nv], z[:, ch + vd + nv:]
    full = torch.cat([(d["tail0"] if case["carried"] else d["tail"]).T, qkv])
    mixed = _silu(sum(full[i:i + T] * d["conv"][:, i] for i in range(s["taps"])))
    unit = lambda x: x * torch.rsqrt(x.square().sum(-1, keepdim=True) + 1e-12)  # noqa: E731
    kd = nk * 128
    q = unit(mixed[:, :kd].view(T, nk, 128)).repeat_interleave(nv // nk, 1) * 128 ** -0.5
    k = unit(mixed[:, kd:2 * kd].view(T, nk, 128)).repeat_interleave(nv // nk, 1)
    decay = torch.exp(-d["a_log"].exp() * torch.nn.functional.softplus(a + d["dt_bias"]))
    o, S = _delta_rule(q, k, mixed[:, 2 * kd:].view(T, nv, 128), decay, torch.sigmoid(b), d["state0"] if case["carried"] else d["state"])
    o = (_rms(o, d["gnorm"]).view(T, vd)) * _silu(gate)
    return {"out": o @ d["w_out"].T, "state": S, "tail": full[-(s["taps"] - 1):].T.contiguous()}


def _work_hybrid(case):
    c, T = QWEN35_4B, case["tokens"]
    nv, vd = c.linear_num_value_heads, c.linear_num_value_heads * 128
    ch = 2 * c.linear_num_key_heads * 128 + vd
    w = c.hidden_size * (ch + 2 * vd + 2 * nv)
    return {"bytes": 2 * w + 4 * T * c.hidden_size + 4 * nv * 128 * 128 * 2, "flops": 2 * T * w + 6 * T * nv * 128 * 128}


# ------------------------------------------------------------------ routed experts
def _prepare_experts(case, seed):
    T, W, ff, E, top, mk, lib = case["tokens"], case["width"], case["ff"], case["experts"], case["top"], _Maker(seed), _lib()
    up = 2 * ff if case["act"] else ff
    score, ids = torch.topk(torch.softmax(mk.normal((T, E), dtype=F32), -1), top)
    s = dict(lib=lib, x=mk.normal((T, W)), up=mk.normal((E, up, W), W ** -0.5), down=mk.normal((E, W, ff), ff ** -0.5), ids=ids.to(I32).contiguous(),
             weights=(score / score.sum(-1, keepdim=True)).contiguous(), y=torch.empty(T, W, dtype=F32, device="cuda"))
    if T >= GROUPED_FROM:
        s["work"] = torch.empty(lib.pk_moe_grouped_workspace_bytes(T, top, E, W, ff), dtype=torch.uint8, device="cuda")
    else:
        s["hid"] = torch.empty(T, top, ff, dtype=BF16, device="cuda")
    return s


def _run_experts(case, s):
    lib, T, W, ff, E, top, act, st = s["lib"], case["tokens"], case["width"], case["ff"], case["experts"], case["top"], case["act"], _stream()
    p = {k: v.data_ptr() for k, v in s.items() if isinstance(v, torch.Tensor)}
    if T >= GROUPED_FROM:
        _ok(lib.pk_moe_grouped_act_p(p["x"], p["up"], p["down"], p["ids"], p["weights"], None, None, p["y"], p["work"], T, top, E, W, ff, act, 0.0, 0.0, st))
    else:
        _ok(lib.pk_moe_up_act_p(p["x"], p["up"], p["ids"], p["hid"], T, top, W, ff, act, 0.0, 0.0, 0, st))
        _ok(lib.pk_moe_down_combine(p["hid"], p["down"], p["ids"], p["weights"], None, None, p["y"], T, top, W, ff, 0, st))
    return s["y"]


def _exact_experts(case, seed):
    s = _prepare_experts(case, seed)
    x, y = s["x"].to(F64), torch.zeros(case["tokens"], case["width"], dtype=F64, device="cuda")
    for e in range(case["experts"]):
        t, k = (s["ids"] == e).nonzero(as_tuple=True)
        if len(t):
            z = x[t] @ s["up"][e].to(F64).T
            h = _silu(z[:, 0::2]) * z[:, 1::2] if case["act"] else torch.relu(z).square()
            y.index_add_(0, t, (h @ s["down"][e].to(F64).T) * s["weights"][t, k].to(F64)[:, None])
    return y


def _work_experts(case):
    T, W, ff, E, top = case["tokens"], case["width"], case["ff"], case["experts"], case["top"]
    per = W * ff * (3 if case["act"] else 2)
    used = E * (1 - (1 - top / E) ** T)  # experts that some token picks
    return {"bytes": 2 * per * used + 6 * T * W, "flops": 2 * T * top * per}


# ------------------------------------------------------------------ attention of the layer-list designs
def _paged_rows(mk, lens, had):
    pages, n_pages = _pages(mk, [a + b for a, b in zip(lens, had)])
    off = [0]
    for pg in pages:
        off.append(off[-1] + len(pg))
    return pages, n_pages, dict(positions=_ints([h + t for h, m in zip(had, lens) for t in range(m)]),
                                req=_ints([i for i, m in enumerate(lens) for _ in range(m)]), off=_ints(off[:-1]), pages=_ints([x for pg in pages for x in pg]))


def _prepare_gqa(case, seed):
    mk, (lens, had) = _Maker(seed), _rows(case)
    H, G, D, dt = case["heads"], case["kv_heads"], case["dim"], F32 if case["f32"] else BF16
    T = sum(lens)
    page_list, n_pages, s = _paged_rows(mk, lens, had)
    ld = (H + 2 * G) * D + (H * D if case["gated"] else 0)
    cache = torch.zeros(n_pages, PAGE, 2 * G * D, dtype=dt, device="cuda")
    for pg, h in zip(page_list, had):
        if h:
            full = torch.zeros(len(pg) * PAGE, 2 * G * D, dtype=dt, device="cuda")
            full[:h] = mk.normal((h, 2 * G * D), 1.0, dt)
            cache[torch.tensor(pg, device="cuda")] = full.view(len(pg), PAGE, -1)
    s.update(lib=_lib(), T=T, lens=lens, had=had, page_list=page_list, ld=ld, rows=mk.normal((T, ld), 1.0, dt), qn=mk.normal((D,), 0.1, dt, 1.0),
             kn=mk.normal((D,), 0.1, dt, 1.0), sink=mk.normal((H,), 1.0, dt), cache=cache, q=torch.empty(T, H * D, dtype=dt, device="cuda"),
             out=torch.empty(T, H * D, dtype=dt, device="cuda"), freq=(500000.0 ** (-torch.arange(0, D // 2, 2, dtype=F32, device="cuda") / (D // 2))))
    return s


def _run_gqa(case, s):
    lib, T, H, G, D, f32, st = s["lib"], s["T"], case["heads"], case["kv_heads"], case["dim"], int(case["f32"]), _stream()
    p = {k: v.data_ptr() for k, v in s.items() if isinstance(v, torch.Tensor)}
    stride = PAGE * 2 * G * D
    prep = ffi.QkPrep(norm_kind=1, q_weight=p["qn"], k_weight=p["kn"], eps=EPS)
    _ok(lib.pk_gqa_norm_append(p["rows"], s["ld"], p["positions"], p["req"], p["off"], p["pages"], p["q"], p["cache"], stride, PAGE, H, G, D, D, D // 2, 0,
                               p["freq"], 1.0, C.byref(prep), T, f32, st))
    gate = p["rows"] + (H + 2 * G) * D * s["rows"].element_size() if case["gated"] else None
    extra = ffi.AttnExtra(window=case["window"], softcap=case["softcap"], gate=gate, gate_ld=s["ld"], max_kv_len=max(a + b for a, b in zip(s["lens"], s["had"])))
    _ok(lib.pk_gqa_attention_ex(p["q"], p["cache"], p["sink"], p["positions"], p["req"], p["off"], p["pages"], p["out"], stride, PAGE, T, H, G, D, D,
                                D ** -0.5, 0, C.byref(extra), f32, st))
    return {"out": s["out"], "cache": s["cache"]}


def _softmax_sink(score, sink):
    """softmax over the last axis with exp(sink) added to the denominator"""
    top = torch.maximum(score.amax(-1, keepdim=True), sink)
    e = torch.exp(score - top)
    return e / (e.sum(-1, keepdim=True) + torch.exp(sink - top))


def _exact_gqa(case, seed):
    s = _prepare_gqa(case, seed)
    T, H, G, D = s["T"], case["heads"], case["kv_heads"], case["dim"]
    rows, cache, pos = s["rows"].to(F64), s["cache"].to(F64), s["positions"].long()
    ang = (pos.to(F32)[:, None] * s["freq"]).to(F64)
    cos, sin = torch.cat([ang.cos()] * 2, 1), torch.cat([ang.sin()] * 2, 1)
    half = D // 2
    rot = lambda x: torch.cat([_rope_half(x[..., :half], cos, sin), x[..., half:]], -1)  # noqa: E731
    q = rot(_rms(rows[:, :H * D].view(T, H, D), s["qn"].to(F64)))
    k = rot(_rms(rows[:, H * D:(H + G) * D].view(T, G, D), s["kn"].to(F64)))
    v = rows[:, (H + G) * D:(H + 2 * G) * D]
    out, row = torch.empty(T, H, D, dtype=F64, device="cuda"), 0
    for m, h, pg in zip(s["lens"], s["had"], s["page_list"]):
        page, at = torch.tensor(pg, device="cuda"), torch.arange(h, h + m, device="cuda")
        cache[page[at // PAGE], at % PAGE] = torch.cat([k[row:row + m].reshape(m, -1), v[row:row + m]], 1)
        kv = cache[page].reshape(-1, 2, G, D)[:h + m]
        j = torch.arange(h + m, device="cuda")
        hidden = (j[None] > at[:, None]) | ((j[None] <= at[:, None] - case["window"]) if case["window"] else torch.zeros((), dtype=torch.bool, device="cuda"))
        for i in range(H):
            sc = (q[row:row + m, i] @ kv[:, 0, i * G // H].T) * D ** -0.5
            if case["softcap"]:
                sc = case["softcap"] * torch.tanh(sc / case["softcap"])
            out[row:row + m, i] = _softmax_sink(sc.masked_fill(hidden, -math.inf), s["sink"][i].to(F64)) @ kv[:, 1, i * G // H]
        row += m
    out = out.view(T, H * D)
    if case["gated"]:
        out = out * torch.sigmoid(rows[:, (H + 2 * G) * D:])
    return {"out": out, "cache": cache}


def _pairs(case):
    """(query, key) pairs that can see each other, and the cached keys that some query sees"""
    w, pairs, keys = case["window"], 0, 0
    for m, h in zip(*_rows(case)):
        see = [min(h + t + 1, w) if w else h + t + 1 for t in range(m)]
        pairs += sum(see)
        keys += min(h, see[0] - 1)
    return pairs, keys


def _work_gqa(case):
    T, H, G, D, el = case["tokens"], case["heads"], case["kv_heads"], case["dim"], 4 if case["f32"] else 2
    pairs, keys = _pairs(case)
    return {"bytes": el * (T * (H * D * (3 if case["gated"] else 2) + 4 * G * D) + keys * 2 * G * D), "flops": 4 * pairs * H * D}


def _prepare_latent(case, seed):
    mk, (lens, had) = _Maker(seed), _rows(case)
    H, D, T = case["heads"], case["rank"] + case["rot"], sum(lens)
    page_list, n_pages, s = _paged_rows(mk, lens, had)
    s.update(lib=_lib(), T=T, lens=lens, had=had, page_list=page_list, qa=mk.normal((T, H, D), 0.5), cache=mk.normal((n_pages, PAGE, D)),
             out=torch.empty(T, H, case["rank"], dtype=BF16, device="cuda"))
    return s


def _run_latent(case, s):
    p = {k: v.data_ptr() for k, v in s.items() if isinstance(v, torch.Tensor)}
    D = case["rank"] + case["rot"]
    _ok(s["lib"].pk_latent_attention_ex(p["qa"], p["cache"], None, p["positions"], p["req"], p["off"], p["pages"], p["out"], PAGE * D, PAGE, s["T"],
                                        case["heads"], case["rank"], case["rot"], 192 ** -0.5, case["window"],
                                        max(a + b for a, b in zip(s["lens"], s["had"])), 0, _stream()))
    return s["out"]


def _exact_latent(case, seed):
    s = _prepare_latent(case, seed)
    qa, cache, row, out = s["qa"].to(F64), s["cache"].to(F64), 0, []
    for m, h, pg in zip(s["lens"], s["had"], s["page_list"]):
        keys = cache[torch.tensor(pg, device="cuda")].reshape(-1, cache.shape[-1])[:h + m]
        j, at = torch.arange(h + m, device="cuda"), torch.arange(h, h + m, device="cuda")
        hidden = (j[None] > at[:, None]) | ((j[None] <= at[:, None] - case["window"]) if case["window"] else torch.zeros((), dtype=torch.bool, device="cuda"))
        o = [torch.softmax(((qa[row:row + m, i] @ keys.T) * 192 ** -0.5).masked_fill(hidden, -math.inf), -1) @ keys[:, :case["rank"]]
             for i in range(case["heads"])]
        out.append(torch.stack(o, 1))
        row += m
    return torch.cat(out)


def _work_latent(case):
    T, H, rank, D = case["tokens"], case["heads"], case["rank"], case["rank"] + case["rot"]
    pairs, keys = _pairs(case)
    return {"bytes": 2 * (T * H * (D + rank) + (keys + T) * D), "flops": 2 * pairs * H * (D + rank)}


# ------------------------------------------------------------------ gated delta rule of the layer-list designs
def _prepare_delta(case, seed):
    mk, n, T = _Maker(seed), case["requests"], case["tokens"]
    H, G, D, dt = case["heads"], case["kv_heads"], case["dim"], F32 if case["f32"] else BF16
    lens = _share(T, n, "tokens") if T > n else [1] * n
    row0 = [sum(lens[:i]) for i in range(n)]
    ld = 2 * G * D + H * D
    return dict(lib=_lib(), lens=lens, row0=row0, ld=ld, qkv=mk.normal((T, ld), 1.0, dt), z=mk.normal((T, 2 * H), 1.0, F32), a_log=mk.normal((H,), 0.7, F32, -1.0),
                dt_bias=mk.normal((H,), 0.5, F32, -1.0), state0=mk.normal((n, H, D, D), 0.1, F32), state=torch.empty(n, H, D, D, dtype=F32, device="cuda"),
                slots=_ints(list(range(n))), starts=_ints(row0), counts=_ints(lens), out=torch.empty(T, H * D, dtype=F32, device="cuda"))


def _run_delta(case, s):
    p = {k: v.data_ptr() for k, v in s.items() if isinstance(v, torch.Tensor)}
    H, G, D = case["heads"], case["kv_heads"], case["dim"]
    s["state"].copy_(s["state0"])  # the sequences' states before this step
    _ok(s["lib"].pk_gated_delta_seq(p["qkv"], s["ld"], 0, G * D, 2 * G * D, p["z"], 2 * H, 0, H, p["a_log"], p["dt_bias"], p["state"], H * D * D, p["slots"],
                                    p["starts"], p["counts"], p["out"], H, G, D, D, len(s["lens"]), int(case["f32"]), _stream()))
    return {"out": s["out"], "state": s["state"]}


def _exact_delta(case, seed):
    s = _prepare_delta(case, seed)
    H, G, D, T = case["heads"], case["kv_heads"], case["dim"], case["tokens"]
    x, z = s["qkv"].to(F64), s["z"].to(F64)
    unit = lambda t: t * torch.rsqrt(t.square().sum(-1, keepdim=True) + 1e-6)  # noqa: E731
    q = unit(x[:, :G * D].view(T, G, D)).repeat_interleave(H // G, 1) * D ** -0.5
    k = unit(x[:, G * D:2 * G * D].view(T, G, D)).repeat_interleave(H // G, 1)
    decay = torch.exp(-s["a_log"].to(F64).exp() * torch.nn.functional.softplus(z[:, :H] + s["dt_bias"]))
    beta, v = torch.sigmoid(z[:, H:]), x[:, 2 * G * D:].view(T, H, D)
    outs, states = [], []
    for i, (r, m) in enumerate(zip(s["row0"], s["lens"])):
        o, S = _delta_rule(q[r:r + m], k[r:r + m], v[r:r + m], decay[r:r + m], beta[r:r + m], s["state0"][i].to(F64))
        outs.append(o)
        states.append(S)
    return {"out": torch.cat(outs).reshape(T, H * D), "state": torch.stack(states)}


def _work_delta(case):
    T, H, G, D, n = case["tokens"], case["heads"], case["kv_heads"], case["dim"], case["requests"]
    return {"bytes": T * ((2 * G + H) * D * (4 if case["f32"] else 2) + 8 * H + 4 * H * D) + 8 * n * H * D * D, "flops": 6 * T * H * D * D}


# ------------------------------------------------------------------ what is called
def prepare(case, seed):
    s = globals()["_prepare_" + case["kind"]](case, int(seed))
    s["case"] = dict(case)
    return s


def run(state):
    return globals()["_run_" + state["case"]["kind"]](state["case"], state)


def exact(case, seed):
    return globals()["_exact_" + case["kind"]](case, int(seed))


def work(case):
    return globals()["_work_" + case["kind"]](case)


def tolerance(case):
    """Relative errors (2-norm) that another correct implementation at the same precision shows: about four times what the path shows against
    64 bits, bf16 roundings between the steps included."""
    if case["kind"] in ("gqa", "delta") and case["f32"]:
        return {"rel": 2e-5, "max": 1e-3}
    return {"model": {"rel": 0.03, "max": 0.3}, "mlp": {"rel": 0.012, "max": 0.08}, "attention": {"rel": 0.012, "max": 0.08},
            "hybrid": {"rel": 0.02, "max": 0.2}, "experts": {"rel": 0.01, "max": 0.08}, "gqa": {"rel": 0.01, "max": 0.08},
            "latent": {"rel": 0.01, "max": 0.08}, "delta": {"rel": 2e-5, "max": 1e-3}}[case["kind"]]
