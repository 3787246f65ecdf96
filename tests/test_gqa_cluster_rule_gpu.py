"""How many CTAs share a (tile, head)'s keys in grouped-query attention of 64 rows and more, on both sides of the rule, and the rows they leave against 64 bits; with
the longest context unknown (0) none do."""
import ctypes as C

import pytest
import torch

from pegainfer_b200 import ffi
from tests.launch_grids import launches

pytestmark = pytest.mark.gpu
BF16, F64, PAGE = torch.bfloat16, torch.float64, 16


@pytest.fixture(scope="module")
def lib():
    l = ffi.lib()
    l.cuda_set_device(0)
    l.cublas_init()
    return l


@pytest.mark.parametrize("lens,had,H,G,D,known,shares", [
    ([64], [0], 16, 4, 128, False, 1), ([100], [900], 4, 2, 64, False, 1), ([700], [0], 2, 1, 64, False, 1),  # the length unknown
    ([64], [191], 2, 1, 128, True, 1), ([64], [192], 2, 1, 128, True, 8), ([300], [0], 2, 1, 64, True, 1), ([512], [0], 2, 1, 64, True, 8),
    ([200], [119], 16, 4, 64, True, 1), ([200], [120], 16, 4, 64, True, 4), ([512], [0], 16, 4, 128, True, 1),
    ([300, 148], [575, 0], 16, 2, 64, True, 1), ([300, 148], [724, 0], 16, 2, 64, True, 2), ([333] * 3, [0] * 3, 16, 4, 128, True, 1)])
def test_shares_of_the_keys(lib, lens, had, H, G, D, known, shares):
    T, n = sum(lens), len(lens)
    g = torch.Generator(device="cuda").manual_seed(T + H + D)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda").to(BF16)  # noqa: E731
    need = [(a + b + PAGE - 1) // PAGE for a, b in zip(lens, had)]
    order = torch.randperm(sum(need), generator=g, device="cuda").to(torch.int32)
    off = [sum(need[:i]) for i in range(n)]
    cache, q = r(sum(need), PAGE, 2 * G * D), r(T, H * D)
    pos = torch.tensor([b + i for a, b in zip(lens, had) for i in range(a)], dtype=torch.int32, device="cuda")
    req = torch.tensor([i for i, a in enumerate(lens) for _ in range(a)], dtype=torch.int32, device="cuda")
    offs = torch.tensor(off, dtype=torch.int32, device="cuda")
    out = torch.full((T, H * D), float("nan"), dtype=BF16, device="cuda")
    x = ffi.AttnExtra(max_kv_len=max(a + b for a, b in zip(lens, had)) if known else 0)

    def call(stream):
        assert lib.pk_gqa_attention_ex(q.data_ptr(), cache.data_ptr(), None, pos.data_ptr(), req.data_ptr(), offs.data_ptr(), order.data_ptr(), out.data_ptr(),
                                       PAGE * 2 * G * D, PAGE, T, H, G, D, D, D ** -0.5, 0, C.byref(x), 0, stream) == 0
    call(None)
    torch.cuda.synchronize()
    row = 0
    for i, (a, b) in enumerate(zip(lens, had)):
        kv = cache[order[off[i]:off[i] + need[i]].long()].reshape(-1, 2, G, D)[:a + b].to(F64)
        hidden = torch.arange(a + b, device="cuda")[None] > torch.arange(b, b + a, device="cuda")[:, None]
        for h in range(H):
            s = q[row:row + a].view(a, H, D)[:, h].to(F64) @ kv[:, 0, h * G // H].T * D ** -0.5
            o = torch.softmax(s.masked_fill(hidden, float("-inf")), -1) @ kv[:, 1, h * G // H]
            got = out[row:row + a].view(a, H, D)[:, h].to(F64)
            # P rounded to bf16 against a running maximum (2^-8 of each weight, of either sign) and one rounding of the result
            assert (got - o).norm() <= 6e-3 * o.norm() and (got - o).abs().max() <= 2 ** -7 * kv[:, 1].abs().max(), (i, h)
        row += a
    (name, grid), = launches(call)
    assert grid == (H, (T + 63) // 64, shares) and ("cluster" in name) == (shares > 1)
