"""The bucketed experts (csrc/moe_grouped.cu) where their tiles can go wrong: experts with no rows, with rows around 16, 64 and 256 and with several
tiles, output sizes off the 128-row weight tiles, every activation, more pairs than the bucket kernel keeps in registers."""
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


def run(lib, x, up, down, ids, wts, act, p0, p1):
    T, W = x.shape
    E, ff, top = up.shape[0], down.shape[2], ids.shape[1]
    ws = torch.zeros(lib.pk_moe_grouped_workspace_bytes(T, top, E, W, ff), dtype=torch.uint8, device="cuda")
    y = torch.full((T + 1, W), 3.0, device="cuda")
    assert lib.pk_moe_grouped_act_p(x.data_ptr(), up.data_ptr(), down.data_ptr(), ids.data_ptr(), wts.data_ptr(), None, None, y.data_ptr(), ws.data_ptr(), T, top,
                                    E, W, ff, act, p0, p1, None) == 0
    torch.cuda.synchronize()
    assert (y[T] == 3.0).all() and lib.pk_b200_wait_errors() == 0
    return y[:T]


def wanted(x, up, down, ids, wts, act, p0, p1):
    y = torch.zeros(x.shape, dtype=torch.float64, device="cuda")
    for e in range(up.shape[0]):
        t, k = (ids == e).nonzero(as_tuple=True)
        if not len(t):
            continue
        z = x[t].double() @ up[e].double().T
        if act == 0:
            h = torch.relu(z).square()
        elif act == 1:
            h = z[:, 0::2] * torch.sigmoid(z[:, 0::2]) * z[:, 1::2]
        else:
            g, u = z[:, 0::2].clamp(max=p0), z[:, 1::2].clamp(-p0, p0)
            h = g * torch.sigmoid(p1 * g) * (u + 1)
        y.index_add_(0, t, (h.bfloat16().double() @ down[e].double().T) * wts[t, k].double()[:, None])
    return y


@pytest.mark.parametrize("act", [0, 1, 2])
@pytest.mark.parametrize("W,ff", [(64, 64), (40, 24), (264, 136), (512, 72)])
@pytest.mark.parametrize("counts", [[0, 1, 15, 16, 17, 0, 63, 64, 65], [255, 0, 256, 257], [700, 3], [0, 0, 5]])
def test_rows_per_expert(lib, counts, W, ff, act):
    g = torch.Generator(device="cuda").manual_seed(sum(counts) + W + act)
    rn = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    E, T = len(counts), sum(counts)
    order = torch.randperm(T, generator=g, device="cuda")
    ids = torch.cat([torch.full((c,), e, device="cuda") for e, c in enumerate(counts)]).to(torch.int32)[order].view(T, 1).contiguous()
    x, up, down = rn(T, W).bfloat16(), (rn(E, ff * (2 if act else 1), W) * W ** -0.5).bfloat16(), (rn(E, W, ff) * ff ** -0.5).bfloat16()
    wts = torch.rand(T, 1, generator=g, device="cuda")
    got, want = run(lib, x, up, down, ids, wts, act, 1.5, 1.7), wanted(x, up, down, ids, wts, act, 1.5, 1.7)
    # the hidden values may round to the other bf16 neighbour where the fp32 sums differ in their last bits
    assert (got.double() - want).norm() <= 2e-3 * want.norm()


@pytest.mark.parametrize("W", [248, 2040, 2048, 2056, 4104])
@pytest.mark.parametrize("counts", [[0, 1, 15, 5], [300, 12, 500]])
def test_rows_around_what_is_fetched_ahead(lib, counts, W):
    """moe_place_kernel holds the first 2048 entries of a warp's first row while it looks for the row's place"""
    test_rows_per_expert(lib, counts, W, 24, 0)


@pytest.mark.parametrize("T,top,E", [(33, 6, 64), (3000, 6, 64), (700, 2, 1500)])
def test_many_pairs_and_experts(lib, T, top, E):
    g = torch.Generator(device="cuda").manual_seed(T)
    rn = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    W, ff = 64, 32
    ids = torch.topk(rn(T, E), top).indices.to(torch.int32).contiguous()
    x, up, down, wts = rn(T, W).bfloat16(), (rn(E, 2 * ff, W) / 8).bfloat16(), (rn(E, W, ff) / 6).bfloat16(), torch.rand(T, top, generator=g, device="cuda")
    got, want = run(lib, x, up, down, ids, wts, 1, 0.0, 0.0), wanted(x, up, down, ids, wts, 1, 0.0, 0.0)
    assert (got.double() - want).norm() <= 2e-3 * want.norm()
    assert torch.equal(got, run(lib, x, up, down, ids, wts, 1, 0.0, 0.0))  # a row does not depend on its slot


@pytest.mark.parametrize("T,top,E", [(32768, 1, 3), (5462, 6, 64), (5500, 6, 64), (40, 3, 511), (40, 3, 512), (7, 1, 2), (297, 1, 511)])
def test_both_forms_of_placing(lib, T, top, E):
    """pairs and experts on both sides of what moe_place_kernel takes, fewer pairs than CTAs"""
    g = torch.Generator(device="cuda").manual_seed(T + E)
    rn = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    W, ff = 64, 32
    ids = torch.topk(rn(T, E), top).indices.to(torch.int32).contiguous()
    x, up, down, wts = rn(T, W).bfloat16(), (rn(E, 2 * ff, W) / 8).bfloat16(), (rn(E, W, ff) / 6).bfloat16(), torch.rand(T, top, generator=g, device="cuda")
    got, want = run(lib, x, up, down, ids, wts, 1, 0.0, 0.0), wanted(x, up, down, ids, wts, 1, 0.0, 0.0)
    # as above: a hidden value may round to the other bf16 neighbour
    assert (got.double() - want).norm() <= 2e-3 * want.norm()
