"""Appending K / V rows to the pool (csrc/paged_kv.cu), a warp per token: rows of fewer pieces than lanes, of more than a round of them, source rows whose heads
lie apart, tokens that do not fill a CTA; copies, so the same bytes."""
import pytest
import torch

from pegainfer_b200 import ffi

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib():
    l = ffi.lib()
    l.cuda_set_device(0)
    l.cublas_init()
    return l


@pytest.mark.parametrize("lens,nkv,hd,ps,gap", [([1], 8, 128, 16, 0), ([5, 40, 2], 1, 8, 16, 0), ([33, 18], 3, 72, 4, 24), ([130], 16, 128, 16, 0), ([17, 3], 9, 256, 32, 8),
                                                ([3000, 2500], 2, 64, 16, 0), ([9], 2, 24, 3, 16)])
def test_same_bytes(lib, lens, nkv, hd, ps, gap):
    g = torch.Generator(device="cuda").manual_seed(sum(lens) + hd)
    T, sh, need = sum(lens), hd + gap, [(n + ps - 1) // ps for n in lens]
    order = torch.randperm(sum(need) + 2, generator=g, device="cuda").to(torch.int32)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731
    k, v = (torch.randn(T, nkv + 1, sh, generator=g, device="cuda").bfloat16() for _ in range(2))
    kv = torch.full((sum(need) + 2, 3, ps, nkv, hd), 9.0, device="cuda").bfloat16()  # a page: K, something else, V
    want, first, row, plane = kv.clone(), [sum(need[:i]) for i in range(len(need) + 1)], 0, ps * nkv * hd
    for r, n in enumerate(lens):
        at = torch.arange(n, device="cuda")
        page = order[first[r] + at // ps].long()
        want[page, 0, at % ps], want[page, 2, at % ps] = k[row:row + n, :nkv, :hd], v[row:row + n, :nkv, :hd]
        row += n
    assert lib.paged_kv_scatter_cuda(kv.data_ptr(), 0, 2 * plane, order.data_ptr(), i32(first).data_ptr(), None, k.data_ptr(), v.data_ptr(),
                                     i32([r for r, n in enumerate(lens) for _ in range(n)]).data_ptr(), i32([j for n in lens for j in range(n)]).data_ptr(), T, nkv, hd, ps,
                                     3 * plane, (nkv + 1) * sh, sh, None) == 0
    torch.cuda.synchronize()
    assert torch.equal(kv, want)
