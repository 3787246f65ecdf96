"""Products of 2 to 4 tokens (gemv.cu): a row has the same bits whichever rows stand beside it, in a stacked projection, in a call of its own, in a vocabulary shard
of any size."""
import ctypes as C

import pytest
import torch

from pegainfer_b200 import ffi
from tests.test_gemv_rows_gpu import args, lib  # noqa: F401

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


@pytest.mark.parametrize("N", [2, 3, 4])
@pytest.mark.parametrize("K,M,cut", [(2560, 60001, [1, 2048, 30000]), (4096, 24576, [6000, 13000]), (5120, 30001, [5, 3000]), (9728, 5000, [2500]), (1032, 9000, [301]), (600, 3000, [9])])
def test_rows_by_themselves(lib, N, K, M, cut):  # noqa: F811
    g = torch.Generator(device="cuda").manual_seed(M + N)
    W, X = torch.randn(M, K, generator=g, device="cuda").to(BF16), torch.randn(N, K, generator=g, device="cuda").to(BF16)

    def product(w):
        y = torch.zeros(N, len(w), dtype=BF16, device="cuda")
        assert lib.pk_b200_gemv_fused(C.byref(args(w, X, [y], [len(w)], len(w), N, K)), None) == 0
        return y
    ends = [0, *cut, M]
    assert torch.equal(product(W), torch.cat([product(W[i:j]) for i, j in zip(ends, ends[1:])], 1))
