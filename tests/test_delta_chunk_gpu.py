"""The gated delta rule in chunks of 16 tokens (csrc/delta_chunk.cuh) behind pk_gated_delta_seq and pk_b200_gated_delta_rule_prefill_recurrent:
lengths around the chunk and around the token-by-token form, unequal entries in one launch, value sizes that end inside a CTA's columns,
unaligned rows, correlated keys, decays from none to nearly everything, and a NaN that must not reach earlier tokens."""
import pytest
import torch

from pegainfer_b200 import ffi

pytestmark = pytest.mark.gpu
F64 = torch.float64


@pytest.fixture(scope="module")
def lib():
    l = ffi.lib()
    l.cuda_set_device(0)
    l.cublas_init()
    return l


def rule(q, k, v, g, beta, S):
    out = []
    for t in range(len(q)):
        S = S * g[t][:, None, None]
        u = (v[t] - torch.einsum("hdv,hd->hv", S, k[t])) * beta[t][:, None]
        S = S + k[t][:, :, None] * u[:, None]
        out.append(torch.einsum("hdv,hd->hv", S, q[t]))
    return torch.stack(out), S


def unit(x, eps):
    return x * torch.rsqrt(x.square().sum(-1, keepdim=True) + eps)


def inputs(lens, H, G, D, V, alike, rate, ld_extra=0, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed + sum(lens) + D)
    T = sum(lens)
    rn = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    x = rn(T, 2 * G * D + H * V + ld_extra)
    x[:, G * D:2 * G * D] = alike * rn(1, G * D) + (1 - alike) * x[:, G * D:2 * G * D]  # keys that share a direction
    return x.bfloat16(), rn(T, 2 * H), rate + 0.7 * rn(H), 0.5 * rn(H) - 1.0, 0.2 * rn(len(lens), H, D, V)


def wanted(x, z, a_log, dt, S0, lens, H, G, D, V):
    x, z = x.double(), z.double()
    q = unit(x[:, :G * D].view(-1, G, D), 1e-6).repeat_interleave(H // G, 1) * D ** -0.5
    k = unit(x[:, G * D:2 * G * D].view(-1, G, D), 1e-6).repeat_interleave(H // G, 1)
    v = x[:, 2 * G * D:2 * G * D + H * V].view(-1, H, V)
    dec, beta = torch.exp(-a_log.double().exp() * torch.nn.functional.softplus(z[:, :H] + dt)), torch.sigmoid(z[:, H:])
    outs, states, r = [], [], 0
    for i, m in enumerate(lens):
        o, S = rule(q[r:r + m], k[r:r + m], v[r:r + m], dec[r:r + m], beta[r:r + m], S0[i].double())
        outs.append(o)
        states.append(S)
        r += m
    return torch.cat(outs), torch.stack(states)


def launch(lib, x, z, a_log, dt, S0, lens, H, G, D, V):
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731
    state, out = S0.clone(), torch.full((sum(lens) + 1, H * V), 5.0, device="cuda")
    slot, row0, ln = i32(list(range(len(lens)))), i32([sum(lens[:i]) for i in range(len(lens))]), i32(lens)
    assert lib.pk_gated_delta_seq(x.data_ptr(), x.stride(0), 0, G * D, 2 * G * D, z.data_ptr(), 2 * H, 0, H, a_log.data_ptr(), dt.data_ptr(), state.data_ptr(),
                                  H * D * V, slot.data_ptr(), row0.data_ptr(), ln.data_ptr(), out.data_ptr(), H, G, D, V, len(lens), 0, None) == 0
    torch.cuda.synchronize()
    assert (out[-1] == 5.0).all() and lib.pk_b200_wait_errors() == 0
    return out[:-1].view(-1, H, V), state


def off(got, want):
    return ((got.double() - want).norm() / want.norm()).item()


@pytest.mark.parametrize("D,V", [(64, 64), (128, 128), (128, 20), (64, 33)])
@pytest.mark.parametrize("lens", [[1], [4], [5], [15], [16], [17], [33, 4, 1, 16], [300, 7]])
def test_lengths(lib, lens, D, V):
    a = inputs(lens, 4, 2, D, V, 0.0, -1.0)
    (got, gs), (want, ws) = launch(lib, *a, lens, 4, 2, D, V), wanted(*a, lens, 4, 2, D, V)
    # fp32 sums of D products (2^-24 each way) over a state that the decays keep bounded: the token-by-token form shows 1.7e-7
    assert off(got, want) < 6e-7 and off(gs, ws) < 6e-7


@pytest.mark.parametrize("D,V", [(64, 64), (64, 129), (64, 300), (128, 128), (128, 65), (128, 200), (128, 3)])
@pytest.mark.parametrize("lens", [[1, 1, 1, 1, 1, 1], [2, 1, 3, 4], [1, 40, 2], [10, 11, 9], [20, 21, 33], [31, 32, 33, 7, 1, 12]])
@pytest.mark.parametrize("H,G", [(4, 2), (24, 12)])
def test_few_tokens(lib, lens, H, G, D, V):
    """Portions of a few tokens: value columns on both sides of what a CTA takes (one, two and all CTAs of a head), both forms in one call, lengths on both
    sides of the choice for one to many waves of CTAs, unaligned pairs of columns."""
    a = inputs(lens, H, G, D, V, 0.0, -1.0)
    (got, gs), (want, ws) = launch(lib, *a, lens, H, G, D, V), wanted(*a, lens, H, G, D, V)
    assert off(got, want) < 6e-7 and off(gs, ws) < 6e-7


@pytest.mark.parametrize("D,V", [(64, 64), (64, 129), (128, 128), (128, 65)])
def test_a_decoded_tokens_result_does_not_depend_on_the_call(lib, D, V):
    """the same bits alone and beside other requests, whatever the columns to a CTA"""
    lens, H, G = [1, 4, 2, 10, 1, 1, 3, 1, 1, 1, 1, 9], 16, 8
    x, z, a_log, dt, S0 = inputs(lens, H, G, D, V, 0.0, -1.0)
    got, gs = launch(lib, x, z, a_log, dt, S0, lens, H, G, D, V)
    for i, n in enumerate(lens):
        r = sum(lens[:i])
        alone, alone_s = launch(lib, x[r:r + n], z[r:r + n], a_log, dt, S0[i:i + 1], [n], H, G, D, V)
        assert torch.equal(alone, got[r:r + n]) and torch.equal(alone_s[0], gs[i])


@pytest.mark.parametrize("alike", [0.5, 0.9, 1.0])
@pytest.mark.parametrize("rate", [-8.0, -1.0, 2.5])
def test_alike_keys_and_strong_decays(lib, alike, rate):
    lens = [200]
    a = inputs(lens, 4, 4, 128, 128, alike, rate)
    (got, gs), (want, ws) = launch(lib, *a, lens, 4, 4, 128, 128), wanted(*a, lens, 4, 4, 128, 128)
    # keys that share a direction subtract nearly equal sums (as token by token does): a few times the error above
    assert off(got, want) < 4e-6 and off(gs, ws) < 4e-6


def test_unaligned_rows(lib):
    lens = [40, 21]
    a = inputs(lens, 4, 2, 64, 64, 0.0, -1.0, ld_extra=3)
    (got, gs), (want, ws) = launch(lib, *a, lens, 4, 2, 64, 64), wanted(*a, lens, 4, 2, 64, 64)
    assert off(got, want) < 6e-7 and off(gs, ws) < 6e-7


@pytest.mark.parametrize("where", ["k", "q", "v"])
def test_nan_reaches_no_earlier_token(lib, where):
    H, G, D, V, lens, at = 2, 2, 64, 64, [48], 21
    a = inputs(lens, H, G, D, V, 0.0, -1.0)
    want, _ = wanted(*a, lens, H, G, D, V)
    a[0][at, {"q": 3, "k": G * D + 3, "v": 2 * G * D + 3}[where]] = float("nan")
    got, _ = launch(lib, *a, lens, H, G, D, V)
    assert off(got[:at], want[:at]) < 6e-7 and torch.isfinite(got[:, 1]).all()
    bad = torch.isnan(got[:, 0])
    if where == "q":
        assert bad[at].all() and not bad[at + 1:].any()
    elif where == "k":
        assert bad[at:].all()
    else:
        assert bad[at:, 3].all() and not bad[:, 4:].any()


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("T", [2, 16, 17, 130])
def test_hybrid_entry(lib, T, shift):
    nk, nv = 2, 4
    g = torch.Generator(device="cuda").manual_seed(T)
    rn = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    W = (2 * nk + nv) * 128
    qkv = torch.zeros(T * W + 8, device="cuda").bfloat16()[shift:shift + T * W].view(T, W)
    qkv.copy_(rn(T, W))
    b, a, dt, a_log, S0 = rn(T, nv).bfloat16(), rn(T, nv).bfloat16(), rn(nv).bfloat16(), 0.5 * rn(nv), 0.1 * rn(nv, 128, 128)
    state, out = S0.clone(), torch.zeros(T, nv * 128, device="cuda").bfloat16()
    assert lib.pk_b200_gated_delta_rule_prefill_recurrent(qkv.data_ptr(), b.data_ptr(), a.data_ptr(), dt.data_ptr(), a_log.data_ptr(), state.data_ptr(),
                                                          out.data_ptr(), nk, nv, 128, 128, T, None) == 0
    torch.cuda.synchronize()
    x = qkv.double()
    q = unit(x[:, :nk * 128].view(T, nk, 128), 1e-12).repeat_interleave(2, 1) * 128 ** -0.5
    k = unit(x[:, nk * 128:2 * nk * 128].view(T, nk, 128), 1e-12).repeat_interleave(2, 1)
    dec = torch.exp(-a_log.double().exp() * torch.nn.functional.softplus(a.double() + dt.double()))
    o, S = rule(q, k, x[:, 2 * nk * 128:].view(T, nv, 128), dec, torch.sigmoid(b.double()), S0.double())
    assert off(state, S) < 6e-7
    assert ((out.view(T, nv, 128).double() - o).abs() <= o.abs() * 2 ** -8 + o.abs().max() * 1e-5).all()  # one bf16 rounding


@pytest.mark.parametrize("n", [1, 3, 15, 17, 31])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("aligned", [True, False])
def test_rows_behind_the_end_are_never_read(lib, n, D, aligned):
    """the last chunk's missing tokens: zeros, whatever lies behind the portion (here NaN), by asynchronous copies and one by one; after a whole chunk, so
    that the chunk form takes it"""
    H, G, V, lens = 4, 2, D, [32 + n]
    x, z, a_log, dt, S0 = inputs([lens[0] + 16], H, G, D, V, 0.0, -1.0, ld_extra=0 if aligned else 3)
    want, ws = wanted(x[:lens[0]], z[:lens[0]], a_log, dt, S0, lens, H, G, D, V)
    x[lens[0]:] = float("nan")
    z[lens[0]:] = float("nan")
    got, gs = launch(lib, x, z, a_log, dt, S0, lens, H, G, D, V)
    assert off(got, want) < 6e-7 and off(gs, ws) < 6e-7
