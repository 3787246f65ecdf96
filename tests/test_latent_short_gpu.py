"""The latent attention of a few tokens with short contexts (csrc/latent_attention_mma.cu): a tile per token where contexts hold two blocks of keys at most,
and two blocks cut or not, on both sides of either rule; tokens of several requests, heads that fill a tile's rows and heads that do not."""
import pytest

from tests.test_latent_tc_gpu import check_against_64_bits, lib  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rank,rot", [(512, 64), (256, 32), (64, 16), (320, 0)])
@pytest.mark.parametrize("starts,lens,H,window,ps,sink", [
    ([77] * 6, [1] * 6, 8, 0, 16, True), ([127, 3, 64], [1, 2, 1], 5, 0, 16, False), ([128, 3], [1, 5], 5, 0, 16, True), ([0, 20, 100], [60, 3, 28], 3, 0, 8, False),
    ([30] * 148, [1] * 148, 2, 0, 16, False), ([30] * 149, [1] * 149, 2, 0, 16, True), ([100] * 37, [1] * 37, 16, 0, 16, False), ([100] * 38, [1] * 38, 16, 0, 16, False), ([64] * 5, [1] * 5, 16, 0, 16, False),
    ([900, 5, 40], [2, 3, 1], 7, 90, 16, False), ([100] * 20, [1] * 20, 33, 0, 16, True)])
def test_against_64_bits(lib, starts, lens, H, window, ps, sink, rank, rot):  # noqa: F811
    check_against_64_bits(lib, starts, lens, H, window, ps, sink, rank, rot)
