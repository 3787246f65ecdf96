"""The bucketed experts where their weights are the first to leave L2 (csrc/moe_grouped.cu), next to the calls on the other side of that rule: one token fewer
than 24 rows an expert, and as many rows as a tile holds.  The same bits for a token in both, and near 64 bits."""
import pytest
import torch

from tests.test_moe_grouped_gpu import lib, run, wanted  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("act,E,W,ff,top", [(0, 24, 2048, 1400, 3), (1, 16, 2048, 1408, 2), (2, 24, 1536, 1240, 4)])
def test_both_sides(lib, act, E, W, ff, top):  # noqa: F811
    assert E * W * ff * (6 if act else 4) > 256 << 20
    g = torch.Generator(device="cuda").manual_seed(W + act)
    rn = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    few, most = 24 * E // top, 240 * E // top
    x, up, down = rn(most + 1, W).bfloat16(), (rn(E, ff * (2 if act else 1), W) * W ** -0.5).bfloat16(), (rn(E, W, ff) * ff ** -0.5).bfloat16()
    wts, ids = torch.topk(torch.softmax(rn(most + 1, E), -1), top)
    wts, ids = wts.contiguous(), ids.to(torch.int32).contiguous()
    part = lambda n: run(lib, x[:n].contiguous(), up, down, ids[:n].contiguous(), wts[:n].contiguous(), act, 1.5, 1.7)  # noqa: E731
    a, b, c, d = part(few - 1), part(few), part(most), part(most + 1)
    assert torch.equal(a, b[:few - 1]) and torch.equal(b, c[:few]) and torch.equal(c, d[:most])
    want = wanted(x, up, down, ids, wts, act, 1.5, 1.7)
    # hidden values are rounded to bf16 (2^-9 relative at most) in both; where fp32 sums put one on the other side, the result moves by a part of a rounding
    assert (d.double() - want).norm() <= 2 ** -9 * want.norm()
