"""The latent attention of prompt portions where its CTAs go on with the grid's next ones: several tiles a CTA, more runs that start inside tiles than its
queue has places, runs of one block and of many in turn, and halves of unequal width, whose CTAs do not.  And few rows with short contexts."""
import pytest
import torch

from tests.test_latent_tc_gpu import check_against_64_bits, lib  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rank,rot", [(512, 64), (256, 32), (384, 48)])
@pytest.mark.parametrize("starts,lens,H,window,ps,sink", [
    ([0], [3333], 16, 0, 16, False), ([50] * 600, [5] * 600, 10, 0, 16, True), ([0, 2000, 5], [1500, 700, 900], 16, 300, 32, True),
    ([3000, 0] * 12, [1, 130] * 12, 16, 0, 16, False), ([0] * 300, [9] * 300, 24, 0, 8, False)])
def test_against_64_bits(lib, starts, lens, H, window, ps, sink, rank, rot):  # noqa: F811
    check_against_64_bits(lib, starts, lens, H, window, ps, sink, rank, rot)


# on both sides of the rule that takes few rows with short contexts here: 12 CTAs (one in twelve SMs) or not, contexts of 64, 128, 129, 512 and 513 keys
@pytest.mark.parametrize("rank,rot", [(512, 64), (256, 32), (128, 32), (64, 16), (320, 0)])
@pytest.mark.parametrize("starts,lens,H,window,ps,sink", [
    ([0], [64], 16, 0, 16, False), ([0], [128], 16, 0, 16, True), ([0, 28], [60, 101], 16, 0, 16, False), ([412], [100], 16, 0, 16, True), ([413], [100], 16, 0, 16, False),
    ([0], [512], 8, 0, 32, False), ([900], [100], 16, 300, 16, False), ([3, 511, 60, 0] * 25, [1] * 100, 20, 0, 16, True), ([0], [90], 16, 0, 16, False)])
def test_few_rows(lib, starts, lens, H, window, ps, sink, rank, rot):  # noqa: F811
    check_against_64_bits(lib, starts, lens, H, window, ps, sink, rank, rot)


def test_captured(lib):  # noqa: F811
    """a captured launch gives the same bits, again and again"""
    T, H, rank, rot, ps = 2000, 16, 512, 64, 16
    D = rank + rot
    g = torch.Generator(device="cuda").manual_seed(1)
    cache, qa = (torch.randn(T, n, generator=g, device="cuda").bfloat16() for n in (D, H * D))
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731
    pos, req, off, pages = i32(list(range(T))), i32([0] * T), i32([0]), i32(list(range(T // ps)))
    out = torch.zeros(T, H, rank, device="cuda").bfloat16()

    def run(st):
        assert lib.pk_latent_attention_ex(qa.data_ptr(), cache.data_ptr(), None, pos.data_ptr(), req.data_ptr(), off.data_ptr(), pages.data_ptr(), out.data_ptr(),
                                          ps * D, ps, T, H, rank, rot, D ** -0.5, 0, T, 0, st) == 0

    run(None)
    torch.cuda.synchronize()
    want, graph, side = out.clone(), torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(graph, stream=side):
        run(torch.cuda.current_stream().cuda_stream)
        run(torch.cuda.current_stream().cuda_stream)
    for _ in range(3):
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want)
    assert lib.pk_b200_wait_errors() == 0
