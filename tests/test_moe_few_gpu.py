"""The experts' products for a few tokens (moe_few.cu) against 64 bits, at the edges of its chunks, units and entries: rows that end inside a block of 64
elements and inside a unit of 16, experts with more than 8 and more than 16 pairs, one and several rounds of units, the last number of pairs that it takes
and the first that it leaves to moe.cu."""
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


def P(t):
    return t.data_ptr() if t is not None else None


@pytest.mark.parametrize("T,top,E,W,ff,act,shared", [
    (1, 1, 1, 8, 8, 0, 0), (1, 6, 64, 2048, 1408, 1, 0), (5, 3, 4, 40, 24, 2, 1), (13, 2, 6, 1032, 200, 0, 2), (31, 6, 64, 136, 72, 1, 1),
    (40, 1, 2, 2056, 16, 0, 0), (96, 2, 3, 72, 1032, 1, 2), (97, 2, 3, 72, 104, 1, 0), (17, 1, 1, 1024, 3000, 2, 0), (4, 2, 16, 3008, 24, 0, 0)])
def test_against_64_bits(lib, T, top, E, W, ff, act, shared):
    g = torch.Generator(device="cuda").manual_seed(T * 1000 + W)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    x, up, down = r(T, W).to(BF16), (r(E, 2 * ff if act else ff, W) * W ** -0.5).to(BF16), (r(E, W, ff) * ff ** -0.5).to(BF16)
    score = r(T, E)
    score[:, 0] += 2.0  # a crowded expert
    w, ids = torch.topk(torch.softmax(score, -1), top)
    w, ids = w.contiguous(), ids.to(torch.int32).contiguous()
    sh, sg = (r(T, W).to(BF16) if shared else None), (r(T) if shared == 2 else None)
    hid, y = torch.zeros(T, top, ff, dtype=BF16, device="cuda"), torch.full((T, W), float("nan"), device="cuda")
    limit, slope = 1.5, 1.7
    assert lib.pk_moe_up_act_p(P(x), P(up), P(ids), P(hid), T, top, W, ff, act, limit, slope, 0, None) == 0
    assert lib.pk_moe_down_combine(P(hid), P(down), P(ids), P(w), P(sh), P(sg), P(y), T, top, W, ff, 0, None) == 0
    torch.cuda.synchronize()
    z = torch.einsum("tkfw,tw->tkf", up.to(F64)[ids.long()], x.to(F64))
    if act == 0:
        want = torch.relu(z).square()
    else:
        a, b = z[..., 0::2], z[..., 1::2]
        if act == 2:
            a, b = a.clamp(max=limit), b.clamp(-limit, limit)
            want = a * torch.sigmoid(slope * a) * (b + 1)
        else:
            want = a * torch.sigmoid(a) * b
    # one rounding to bf16 (2^-9 relative) beside fp32 sums (1e-6 of the row's products)
    assert ((hid.to(F64) - want).abs() <= want.abs() * 2 ** -8 + 2e-5).all()
    out = (torch.einsum("tkwf,tkf->tkw", down.to(F64)[ids.long()], hid.to(F64)) * w.to(F64)[..., None]).sum(1)
    if shared:
        out = out + sh.to(F64) * (torch.sigmoid(sg.to(F64))[:, None] if shared == 2 else 1.0)
    assert ((y.to(F64) - out).abs() <= 2e-5 * (1 + out.abs())).all()  # fp32 sums
    assert lib.pk_b200_wait_errors() == 0


def test_a_tokens_result_does_not_depend_on_the_others(lib):
    """and what another token holds (a NaN) stays in its own rows"""
    T, top, E, W, ff = 24, 2, 4, 264, 136
    g = torch.Generator(device="cuda").manual_seed(3)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    x, up, down = r(T, W).to(BF16), (r(E, 2 * ff, W) * W ** -0.5).to(BF16), (r(E, W, ff) * ff ** -0.5).to(BF16)
    w, ids = torch.topk(torch.softmax(r(T, E), -1), top)
    w, ids = w.contiguous(), ids.to(torch.int32).contiguous()

    def run(rows, x):
        n = len(rows)
        i, ww, xx = ids[rows].contiguous(), w[rows].contiguous(), x[rows].contiguous()
        hid, y = torch.zeros(n, top, ff, dtype=BF16, device="cuda"), torch.zeros(n, W, device="cuda")
        assert lib.pk_moe_up_act_p(P(xx), P(up), P(i), P(hid), n, top, W, ff, 1, 0.0, 0.0, 0, None) == 0
        assert lib.pk_moe_down_combine(P(hid), P(down), P(i), P(ww), None, None, P(y), n, top, W, ff, 0, None) == 0
        torch.cuda.synchronize()
        return y

    whole = run(list(range(T)), x)
    assert torch.equal(run([7], x), whole[7:8]) and torch.equal(run([20, 7, 3], x), whole[[20, 7, 3]])
    bad = x.clone()
    bad[5] = float("nan")
    got = run(list(range(T)), bad)
    assert torch.isnan(got[5]).all() and torch.equal(got[[i for i in range(T) if i != 5]], whole[[i for i in range(T) if i != 5]])
