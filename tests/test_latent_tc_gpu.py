"""The latent attention of prompt portions on tcgen05 (csrc/latent_attention_tc.cu): tiles that several requests share, windows, contexts carried over,
page sizes on both sides of a key block, feature counts off its 64-wide chunks, and caches whose unused slots hold NaN."""
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


@pytest.mark.parametrize("rank,rot", [(512, 64), (256, 32), (64, 8), (320, 0)])
@pytest.mark.parametrize("starts,lens,H,window,ps,sink", [
    ([0], [700], 16, 0, 16, False), ([0, 130, 5], [300, 333, 67], 16, 0, 16, True), ([500, 0], [400, 301], 16, 150, 8, True),
    ([40], [1300], 8, 64, 32, False), ([0] * 40, [17 + i for i in range(40)], 10, 0, 128, True), ([3, 900], [640, 1], 16, 1000, 64, False)])
def test_against_64_bits(lib, starts, lens, H, window, ps, sink, rank, rot):
    check_against_64_bits(lib, starts, lens, H, window, ps, sink, rank, rot)


# other chunks of a CTA from none to eight, value chunks from one to four, and both in one launch.  Rings of 0, 2, 6 and 8 places (two blocks' other
# chunks) and of 9, which is less than two blocks' from five other chunks on: 448 + 64, 384 + 48 (one of the halves), 512 + 16 and the last three
@pytest.mark.parametrize("rank,rot", [(256, 0), (64, 64), (448, 64), (384, 48), (512, 16), (192, 384), (128, 448), (64, 512)])
@pytest.mark.parametrize("starts,lens,H,window,ps,sink", [([0, 77], [900, 301], 16, 0, 16, True), ([300, 0, 9], [1, 700, 340], 16, 130, 128, False)])
def test_places_for_chunks(lib, starts, lens, H, window, ps, sink, rank, rot):
    check_against_64_bits(lib, starts, lens, H, window, ps, sink, rank, rot)


def check_against_64_bits(lib, starts, lens, H, window, ps, sink, rank, rot):
    D, T = rank + rot, sum(lens)
    g = torch.Generator(device="cuda").manual_seed(T + rank)
    rn = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    need = [(s + n + ps - 1) // ps for s, n in zip(starts, lens)]
    order = torch.randperm(sum(need) + 3, generator=g, device="cuda").tolist()
    stride = ps * D + 24
    cache = torch.full((sum(need) + 3, stride), float("nan"), device="cuda").bfloat16()
    off, k = [], 0
    ctx = []
    for s, n, m in zip(starts, lens, need):
        rows = rn(s + n, D).bfloat16()
        rows[:, 0] += 1.0
        ctx.append(rows)
        for p in range(m):
            part = rows[p * ps:(p + 1) * ps]
            cache[order[k + p], :len(part) * D] = part.reshape(-1)
        off.append(k)
        k += m
    qa, sk = (1.5 * rn(T, H, D)).bfloat16(), rn(H).bfloat16()
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731
    pos = i32([s + j for s, n in zip(starts, lens) for j in range(n)])
    req = i32([r for r, n in enumerate(lens) for _ in range(n)])
    out = torch.full((T + 1, H, rank), 9.0, device="cuda").bfloat16()
    off_d, pages_d, scale = i32(off), i32(order), 1.3 * D ** -0.5
    assert lib.pk_latent_attention_ex(qa.data_ptr(), cache.data_ptr(), sk.data_ptr() if sink else None, pos.data_ptr(), req.data_ptr(), off_d.data_ptr(),
                                      pages_d.data_ptr(), out.data_ptr(), stride, ps, T, H, rank, rot, scale, window,
                                      max(s + n for s, n in zip(starts, lens)), 0, None) == 0
    torch.cuda.synchronize()
    assert (out[T] == 9.0).all() and lib.pk_b200_wait_errors() == 0
    row = 0
    for s, n, keys in zip(starts, lens, ctx):
        kd = keys.double()
        at, j = torch.arange(s, s + n, device="cuda")[:, None], torch.arange(s + n, device="cuda")[None]
        hidden = (j > at) | ((j <= at - window) if window else (j < 0))
        for h in range(H):
            sc = (qa[row:row + n, h].double() @ kd.T * scale).masked_fill(hidden, -float("inf"))
            if sink:
                sc = torch.cat([sc, sk[h].double().expand(n, 1)], 1)
            p = torch.softmax(sc, -1)[:, :s + n]
            want, got = p @ kd[:, :rank], out[row:row + n, h].double()
            # weights and result are rounded to bf16 once each; a row's weights are positive, so the first rounding stays below 2^-8 of |v| weighed
            bound = 2 ** -8 * (p @ kd[:, :rank].abs()) + 2 ** -8 * want.abs() + 1e-4
            assert ((got - want).abs() <= bound).all(), (h, (got - want).abs().max().item())
        row += n


@pytest.mark.parametrize("spread", [0.9, 4.0, 8.0])
def test_as_near_to_64_bits_as_the_other_kernel(lib, spread):
    """The same rows through this kernel (one call) and through the mma.sync kernel (calls of 24 tokens, too few for this one).  Both follow the exact
    maximum, so that the largest weight needs no rounding; a reference that lags behind it made peaked scores' errors 1.17 to 1.22 times as large.
    The two errors differ by chance alone: 1.03 leaves ten times what 2^20 outputs of independent roundings show."""
    T, H, rank, rot, ps = 768, 16, 512, 64, 16
    D = rank + rot
    g = torch.Generator(device="cuda").manual_seed(5)
    rn = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    cache, qa = rn(T, D).bfloat16(), (spread * rn(T, H, D)).bfloat16()
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731
    pos, req, off, pages = torch.arange(T, device="cuda", dtype=torch.int32), i32([0] * T), i32([0]), i32(list(range(T // ps)))
    out = torch.zeros(2, T, H, rank, device="cuda").bfloat16()

    def run(to, t0, n):
        assert lib.pk_latent_attention_ex(qa[t0:].data_ptr(), cache.data_ptr(), None, pos[t0:].data_ptr(), req[t0:].data_ptr(), off.data_ptr(), pages.data_ptr(),
                                          out[to, t0:].data_ptr(), ps * D, ps, n, H, rank, rot, D ** -0.5, 0, T, 0, None) == 0

    run(0, 0, T)
    for t0 in range(0, T, 24):
        run(1, t0, 24)
    torch.cuda.synchronize()
    hidden = torch.arange(T, device="cuda")[None] > torch.arange(T, device="cuda")[:, None]
    err = [0.0, 0.0]
    for h in range(H):
        want = torch.softmax((qa[:, h].double() @ cache.double().T * D ** -0.5).masked_fill(hidden, -float("inf")), -1) @ cache[:, :rank].double()
        for i in range(2):
            err[i] += (out[i, :, h].double() - want).square().sum().item()
    assert (err[0] / err[1]) ** 0.5 < 1.03, err


@pytest.mark.parametrize("rank,rot,H", [(64, 8, 8), (128, 24, 8), (576, 0, 8)])
def test_shapes_of_the_generic_kernel_keep_its_weights(lib, rank, rot, H):
    """what the mma.sync kernel does not take (rot off 16, rank above 512) runs with fp32 weights however many the tokens: only the result is rounded"""
    T, ps, D = 1300, 16, rank + rot
    g = torch.Generator(device="cuda").manual_seed(D)
    rn = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    need = (T + ps - 1) // ps
    cache, qa = torch.zeros(need * ps, D, device="cuda").bfloat16(), (2 * rn(T, H, D)).bfloat16()
    cache[:T] = rn(T, D).bfloat16()
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731
    pos, req, off, pages = torch.arange(T, device="cuda", dtype=torch.int32), i32([0] * T), i32([0]), i32(list(range(need)))
    out = torch.zeros(T, H, rank, device="cuda").bfloat16()
    assert lib.pk_latent_attention_ex(qa.data_ptr(), cache.data_ptr(), None, pos.data_ptr(), req.data_ptr(), off.data_ptr(), pages.data_ptr(), out.data_ptr(),
                                      ps * D, ps, T, H, rank, rot, D ** -0.5, 0, T, 0, None) == 0
    torch.cuda.synchronize()
    hidden = torch.arange(T, device="cuda")[None] > torch.arange(T, device="cuda")[:, None]
    kd = cache[:T].double()
    for h in range(H):
        p = torch.softmax((qa[:, h].double() @ kd.T * D ** -0.5).masked_fill(hidden, -float("inf")), -1)
        want, size = p @ kd[:, :rank], p @ kd[:, :rank].abs()
        # scores of a few units from fp32 sums of D products: a weight is off by 2^-18 at most, and so is the sum
        assert ((out[:, h].double() - want).abs() <= want.abs() * 2 ** -8 + size * 2 ** -16).all()


@pytest.mark.parametrize("H,ps", [(16, 16), (10, 64)])
@pytest.mark.parametrize("sink", [False, True])
def test_what_another_requests_cache_holds_stays_there(lib, H, ps, sink):
    """a request whose visible keys are NaN beside others in the same 128-row tiles: their rows are those of a call where it is sound"""
    rank, rot, lens = 512, 64, [290, 3, 309]
    D, T = rank + rot, sum(lens)
    g = torch.Generator(device="cuda").manual_seed(H)
    rn = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    need = [(n + ps - 1) // ps for n in lens]
    cache, qa, sk = rn(sum(need) * ps, D).bfloat16(), rn(T, H, D).bfloat16(), rn(H).bfloat16()
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731
    off = [sum(need[:i]) for i in range(3)]
    pos, req = i32([j for n in lens for j in range(n)]), i32([r for r, n in enumerate(lens) for _ in range(n)])
    off_d, pages = i32(off), i32(list(range(sum(need))))

    def run(c):
        out = torch.zeros(T, H, rank, device="cuda").bfloat16()
        assert lib.pk_latent_attention_ex(qa.data_ptr(), c.data_ptr(), sk.data_ptr() if sink else None, pos.data_ptr(), req.data_ptr(), off_d.data_ptr(),
                                          pages.data_ptr(), out.data_ptr(), ps * D, ps, T, H, rank, rot, D ** -0.5, 0, max(lens), 0, None) == 0
        torch.cuda.synchronize()
        return out

    sound = run(cache)
    assert torch.isfinite(sound).all()
    for bad in range(3):
        c = cache.clone()
        c[off[bad] * ps:(off[bad] + need[bad]) * ps, :64] = float("nan")
        got, row = run(c), 0
        for r, n in enumerate(lens):
            if r != bad:
                assert torch.equal(got[row:row + n], sound[row:row + n]), (bad, r)
            else:
                assert torch.isnan(got[row:row + n, :, :64]).all()
            row += n


def test_rows_without_a_visible_key(lib):
    """positions before the first key, whole tiles of them and some beside others: a row of zeros with a sink (the other kernels' result)"""
    T, H, rank, rot, ps = 600, 16, 512, 64, 16
    D = rank + rot
    g = torch.Generator(device="cuda").manual_seed(1)
    rn = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    cache, qa, sk = rn(304 * ps, D).bfloat16(), rn(T, H, D).bfloat16(), rn(H).bfloat16()
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731
    pos, req = i32([-1] * 300 + list(range(300))), i32([0] * 300 + [1] * 300)
    off, pages, out = i32([0, 2]), i32(list(range(304))), torch.full((T, H, rank), 3.0, device="cuda").bfloat16()
    assert lib.pk_latent_attention_ex(qa.data_ptr(), cache.data_ptr(), sk.data_ptr(), pos.data_ptr(), req.data_ptr(), off.data_ptr(), pages.data_ptr(),
                                      out.data_ptr(), ps * D, ps, T, H, rank, rot, D ** -0.5, 0, 300, 0, None) == 0
    torch.cuda.synchronize()
    assert (out[:300] == 0).all() and torch.isfinite(out[300:]).all() and (out[300:] != 0).any(-1).all() and lib.pk_b200_wait_errors() == 0


@pytest.mark.parametrize("starts,lens,H,window,ps,sink", [
    ([0] + [60 * i + 5 for i in range(20)], [500] + [1] * 20, 16, 0, 16, True),            # a portion and decoded tokens behind it
    ([40 * i for i in range(13)] + [100, 0], [1] * 13 + [290, 4], 16, 70, 8, False),      # in front of it, windows; odd rests
    ([(7 * i) % 400 for i in range(300)], [1] * 300, 16, 0, 64, True),                    # decoded tokens alone
    ([3, 500, 0, 77, 9, 1], [20, 1, 1, 30, 2, 1], 100, 0, 16, False),                     # tokens across the borders of tiles
    ([3, 0, 77, 9], [17, 1, 20, 2], 128, 0, 16, True), ([3, 0, 77], [8, 1, 11], 256, 0, 16, False),  # tokens that fill whole tiles
    ([i % 5 for i in range(9600)], [1] * 9600, 1, 0, 8, False)])                          # more runs than the helpers of one GPU's SMs list
def test_many_requests_in_a_tile(lib, starts, lens, H, window, ps, sink):
    test_against_64_bits(lib, starts, lens, H, window, ps, sink, 512, 64)
