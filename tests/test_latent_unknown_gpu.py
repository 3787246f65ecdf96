"""Latent attention of calls that do not know their longest context (0): the same rows as with it, in tiles of a token each (fewer than 16 heads) or of 16 rows."""
import pytest

from tests.test_latent_tc_gpu import check_against_64_bits, lib  # noqa: F401

pytestmark = pytest.mark.gpu


class LengthUnknown:
    def __init__(self, lib):
        self.lib = lib

    def __getattr__(self, name):
        return getattr(self.lib, name)

    def pk_latent_attention_ex(self, *args):
        return self.lib.pk_latent_attention_ex(*args[:-3], 0, *args[-2:])


@pytest.mark.parametrize("rank,rot", [(512, 64), (64, 16)])
@pytest.mark.parametrize("starts,lens,H,window", [([900] * 3, [1, 2, 5], 5, 0), ([300, 20], [1, 1], 16, 0), ([500, 2], [3, 4], 4, 90), ([0], [149], 2, 0)])
def test_against_64_bits(lib, starts, lens, H, window, rank, rot):  # noqa: F811
    check_against_64_bits(LengthUnknown(lib), starts, lens, H, window, 16, True, rank, rot)
