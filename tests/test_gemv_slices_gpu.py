"""pk_b200_gemv_slices names the grid that a call of one to four tokens is launched with, whichever kernel takes it."""
import ctypes as C

import pytest
import torch

from pegainfer_b200 import ffi
from tests.launch_grids import launches
from tests.test_gemv_rows_tp_gpu import two_ranks
from tests.test_gemv_rows_gpu import args, lib  # noqa: F401

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


@pytest.mark.parametrize("N", [1, 2, 3, 4])
@pytest.mark.parametrize("M,epi", [(1, 0), (16, 1), (147, 0), (297, 0), (301, 1), (2560, 0), (9728, 1)])
def test_grid_of_the_launch(lib, N, M, epi):  # noqa: F811
    K = 512
    W, X, Y = torch.zeros(2 * M, K, dtype=BF16, device="cuda"), torch.zeros(N, K, dtype=BF16, device="cuda"), torch.zeros(N, M, dtype=BF16, device="cuda")
    comms, stage, flags = two_ranks(lib)
    for x_mode in (0, 1, 2):  # (2: its wait finds the sequence number 0 of a fresh communicator)
        h = torch.zeros_like(X)
        a = args(W, X, [Y], [M], M, N, K, epi=epi, x_mode=x_mode, residual=X, norm_w=X, hidden_out=h if x_mode else None, eps=1e-6, tp_comm=comms[0])

        def call(stream):
            assert lib.pk_b200_gemv_fused(C.byref(a), stream) == 0
        call(None)
        torch.cuda.synchronize()
        (_, grid), = launches(call)
        assert grid == (lib.pk_b200_gemv_slices(M, N, x_mode, epi), 1, 1), x_mode
        if N == 1 or x_mode == 2:
            assert grid[0] == lib.pk_b200_gemv_grid(M, epi)
    assert lib.pk_b200_gemv_slices(0, 1, 0, 0) == 0 and lib.pk_b200_gemv_slices(5, 5, 0, 0) == 0 and lib.pk_b200_wait_errors() == 0
