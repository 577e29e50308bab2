"""The float products and float attention on the tensor cores: operands without three bfloat16 parts, exact products, and the
tiles that the product chooses by its sizes."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(scope="module")
def ops():
    from beglin_b200.csrc import ops as o
    o.lib()
    return o


def rnd(*shape, seed=0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return torch.empty(shape, device=DEV).normal_(generator=g)


def product(ops, a, w, bias=None):
    out = torch.empty((a.shape[0], w.shape[0]), device=DEV)
    ops.gemm_f32_nt(a, w, bias, out)
    return out


@pytest.mark.parametrize("K", [129, 600, 1100])
@pytest.mark.parametrize("M", [3, 40, 200])
def test_operands_without_three_parts(ops, M, K):
    """Infinities, NaN, numbers next to the largest float and below 2^-110, on either side: what floats make of them, row by row."""
    a, w = rnd(M, K, seed=1) * 0.125, rnd(130, K, seed=2) * 0.125
    a[0, 5], a[1, K - 1], a[2, 70] = math.inf, math.nan, 3.4e38
    w[7, 3], w[129, 128] = -math.inf, 3.4e38
    if M > 3:
        a[5] = rnd(K, seed=3) * 1e-38                       # a row of small numbers beside ones of the usual size
        a[6, :] = 0.0
    out, want = product(ops, a, w), a.double() @ w.double().t()
    lost = want.abs() > 3.4028234e38
    same = torch.isnan(out) == torch.isnan(want)
    assert bool((same | lost).all()) and bool((torch.isinf(out) | torch.isnan(out))[lost].all())
    fine = torch.isfinite(want) & ~lost
    # a chain of K rounded sums, and the smallest float for what lies below it
    bound = (K + 8) * 2.0 ** -24 * (a.abs().double() @ w.abs().double().t()) + K * 2.0 ** -149
    assert bool(((out.double() - want).abs() <= bound)[fine].all())
    for m in range(min(M, 8)):
        assert torch.equal(product(ops, a[m:m + 1].contiguous(), w).view(torch.int32), out[m:m + 1].view(torch.int32)), m


def test_small_numbers_keep_their_digits(ops):
    a, w = rnd(20, 300, seed=4) * 1e-38, rnd(70, 300, seed=5) * 1e37
    out, want = product(ops, a, w), a.double() @ w.double().t()
    assert bool(((out.double() - want).abs() <= 308 * 2.0 ** -24 * (a.abs().double() @ w.abs().double().t())).all())


@pytest.mark.parametrize("M,N,K", [(3, 130, 600), (40, 64, 1100), (200, 203, 300)])
def test_powers_of_two_change_no_bit(ops, M, N, K):
    """Small operands are summed as those of the usual size are, all of them or one in a row."""
    a, w = rnd(M, K, seed=16), rnd(N, K, seed=17)
    out = product(ops, a, w)
    assert torch.equal(product(ops, a * 2.0 ** -100, w) * 2.0 ** 100, out) and torch.equal(product(ops, a, w * 2.0 ** -100) * 2.0 ** 100, out)
    assert torch.equal(product(ops, a * 2.0 ** -100, w * 2.0 ** 80) * 2.0 ** 20, out)
    a[:, 70], w[:, 100] = 0.0, 0.0
    out = product(ops, a, w)
    a[:, 70], w[:, 100] = 1e-36, 1e-36
    assert torch.equal(product(ops, a, w), out)


def test_weights_that_the_kernel_before_makes(ops):
    """Weights off 16 bytes are read behind the kernel before, for few rows too."""
    a = rnd(3, 201, seed=18)
    for i in range(4):
        w, made = rnd(64, 201, seed=19 + i), torch.empty(64 * 201 + 1, device=DEV)[1:].view(64, 201)
        ops.gemm_f32_nt(w, torch.eye(201, device=DEV), None, made)
        out = product(ops, a, made)
        torch.cuda.synchronize()
        assert torch.equal(made, w) and torch.equal(out, product(ops, a, made))


def test_single_numbers_come_through_whole(ops):
    w = rnd(200, 300, seed=6)
    assert torch.equal(product(ops, torch.eye(300, device=DEV), w), w.t())


@pytest.mark.parametrize("M,N,K", [(16, 130, 1100), (31, 17920, 200), (64, 9000, 320), (96, 9472, 260), (128, 9472, 200), (143, 18944, 192), (160, 18944, 192),
                                   (300, 9472, 136), (161, 257, 8200)])
def test_tiles_of_all_sizes(ops, M, N, K):
    a, w, b = rnd(M, K, seed=7), rnd(N, K, seed=8), rnd(N, seed=9)
    out = product(ops, a, w, b)
    want = a.double() @ w.double().t() + b.double()
    assert bool(((out.double() - want).abs() <= (K + 8) * 2.0 ** -24 * (a.abs().double() @ w.abs().double().t() + b.abs().double())).all())
    for m in (0, M // 2, M - 1):
        assert torch.equal(product(ops, a[m:m + 1].contiguous(), w, b)[0], out[m]), m


@pytest.mark.parametrize("M", [5, 40, 100, 150])
@pytest.mark.parametrize("N", [1, 15, 130, 203])
def test_features_that_fill_no_warp(ops, M, N):
    """Several ranges, walked and added, whose sums some lanes of a warp do not store: the same bits each time."""
    a, w, b = rnd(M, 4000, seed=13), rnd(N, 4000, seed=14), rnd(N, seed=15)
    out, want = product(ops, a, w, b), a.double() @ w.double().t() + b.double()
    assert bool(((out.double() - want).abs() <= 4008 * 2.0 ** -24 * (a.abs().double() @ w.abs().double().t() + b.abs().double())).all())
    assert all(torch.equal(product(ops, a, w, b), out) for _ in range(5))


@pytest.mark.parametrize("accumulate", [False, True])
def test_ranges_in_several_launches(ops, accumulate):
    """An inner size whose ranges take more than one launch, the last of fewer ranges than the first (146 of 960, 145 at a time).  Whole
    numbers: every sum is exact."""
    M, N, K = 160, 64, 140000
    g = torch.Generator(device=DEV).manual_seed(12)
    a, w = (torch.randint(-1, 2, (n, K), device=DEV, generator=g).float() for n in (M, N))
    old = torch.randint(-99, 100, (M, N), device=DEV, generator=g).float()
    out = old.clone()
    ops.gemm_f32_nt(a, w, None, out, accumulate=accumulate)
    assert torch.equal(out.double(), a.double() @ w.double().t() + (old.double() if accumulate else 0.0))


@pytest.mark.parametrize("hd", [48, 80, 128])
def test_attention_of_queries_without_three_parts(ops, hd):
    """Queries below 2^-110 against keys as large: scores of the usual size, every digit of them needed."""
    n, nh, page = 70, 2, 16
    pages = -(-n // page)
    pool = rnd(pages, 2, 1, page, hd, seed=10)
    pool[:, 0] *= 1e37
    q = rnd(n, nh * hd, seed=11) * 1e-37
    pos = torch.arange(n, dtype=torch.int32, device=DEV)
    _, bq, tile = ops.attention_plan(nh, hd, torch.float32, False, "generic", page)
    blocks = torch.tensor([(0, r, min(bq, n - r)) for r in range(0, n, bq)], dtype=torch.int32, device=DEV)
    out, status = torch.empty((n, nh * hd), device=DEV), ops.new_status(DEV)
    table = torch.arange(pages, dtype=torch.int32, device=DEV).view(1, -1)
    ops.attention(q, nh * hd, pool, table, pos, blocks, len(blocks), n - 1, n, nh, 1, hd, 0, 256, tile, bq, hd ** -0.5, out, status, "generic")
    ops.raise_on_status(status)
    k, v = (pool[:, i, 0].reshape(-1, hd)[:n].double() for i in (0, 1))
    for h in range(nh):
        s = (q[:, h * hd:(h + 1) * hd].double() @ k.t()) * hd ** -0.5
        s = s.masked_fill(torch.triu(torch.ones(n, n, dtype=torch.bool, device=DEV), 1), -math.inf)
        want = torch.softmax(s, -1) @ v
        # a score's error moves a weight by as much: hd + 8 roundings of the largest sum of products
        assert (out[:, h * hd:(h + 1) * hd].double() - want).abs().max() <= (hd + 8) * 2.0 ** -23 * float(s.abs()[s > -math.inf].max() + 1) * float(v.abs().max())


def attend(ops, q, k, v, split=256, window=0, slopes=None, softcap=0.0, keep=0, page=16, scale=None):
    """q [n, heads, features], k and v [n, kv heads, features]: a prompt's rows over themselves, one block table."""
    n, nh, hd = q.shape
    nkv, vd = v.shape[1], v.shape[2]
    pages = -(-n // page)
    pad = lambda t: torch.cat([t, torch.zeros((pages * page - n,) + t.shape[1:], device=DEV)]).view(pages, page, nkv, -1).transpose(1, 2).reshape(pages, -1)
    pool = torch.cat([pad(k), pad(v)], dim=1)
    if vd == hd:
        pool = pool.view(pages, 2, nkv, page, hd)
    pos, table = torch.arange(n, dtype=torch.int32, device=DEV), torch.arange(pages, dtype=torch.int32, device=DEV).view(1, -1)
    _, bq, tile = ops.attention_plan(nh // nkv, hd, torch.float32, False, "generic", page, vd=vd)
    blocks = torch.tensor([(0, r, min(bq, n - r)) for r in range(0, n, bq)], dtype=torch.int32, device=DEV)
    out, status = torch.full((n, nh * vd), -7.0, device=DEV), ops.new_status(DEV)
    ops.attention(q.reshape(n, -1), nh * hd, pool, table, pos, blocks, len(blocks), n - 1, n, nh, nkv, hd, window, split, tile, bq,
                  hd ** -0.5 if scale is None else scale, out, status, "generic", softcap=softcap, vd=vd, keep=keep, slopes=slopes)
    ops.raise_on_status(status)
    return out.view(n, nh, vd)


@pytest.mark.parametrize("nh,nkv,hd,vd,window,keep", [(6, 1, 128, 128, 0, 0), (2, 2, 64, 64, 40, 3), (3, 1, 80, 48, 100, 0)])
@pytest.mark.parametrize("split", [64, 256, 1024])
def test_attention_of_several_values_without_three_parts(ops, nh, nkv, hd, vd, window, keep, split):
    """Infinities and NaN in both halves of tiles one behind the other: they reach the rows that see them, and the same ones each time."""
    n, bad_at = 330, [3, 40, 61, 70, 97, 99, 127, 128, 200, 255, 256, 300]
    q, k, v = rnd(n, nh, hd, seed=20), rnd(n, nkv, hd, seed=21), rnd(n, nkv, vd, seed=22)
    v[bad_at, :, 1] = 0.25
    fine = attend(ops, q, k, v, split, window, keep=keep)
    for i, at in enumerate(bad_at):
        v[at, :, 1] = (math.inf, math.nan, -math.inf)[i % 3]
    pos = torch.arange(n, device=DEV)[:, None]
    at = torch.tensor(bad_at, device=DEV)[None, :]
    sees = ((at <= pos) & ((at > pos - window) if window else (at >= 0)) | ((at < keep) & (at <= pos))).any(1)
    other = torch.arange(vd, device=DEV) != 1
    for _ in range(8):
        out = attend(ops, q, k, v, split, window, keep=keep)
        assert torch.isfinite(fine).all() and torch.equal(out[~sees], fine[~sees]) and torch.equal(out[..., other], fine[..., other])
        assert not torch.isfinite(out[sees][..., 1]).any()


@pytest.mark.parametrize("size", [1e20, 1e36])
@pytest.mark.parametrize("hd", [64, 128])
def test_attention_of_small_weights_beside_large_values(ops, hd, size):
    """Weights down to the smallest float, which large values make count: a key's share is off by a few roundings of the weight."""
    n = 50
    q, k, v = torch.zeros((n, 1, hd), device=DEV), torch.zeros((n, 1, hd), device=DEV), rnd(n, 1, hd, seed=30) * size
    away = torch.linspace(70, 103, n, device=DEV).mul(8).round().div(8)
    away[0], v[0] = 0.0, 0.0
    q[:, :, 0], k[:, 0, 0] = 1.0, -8.0 * away
    out = attend(ops, q, k, v, scale=0.125)[-1, 0].double()
    w = torch.exp(-away.double())
    bound = (w * 2.0 ** -21 + 2.0 ** -149) @ v[:, 0].abs().double() + n * 2.0 ** -24 * (w @ v[:, 0].abs().double())
    assert bool(((out * w.sum() - w @ v[:, 0].double()).abs() <= bound).all())
    v[40, 0, 5] = math.inf                                 # a weight of some 1e-42 is not nought
    out = attend(ops, q, k, v, scale=0.125)
    assert away[40] > 96 and torch.isinf(out[40:, 0, 5]).all() and torch.isfinite(out[:40]).all()


@pytest.mark.parametrize("hd", [48, 80, 128])
def test_attention_of_small_operands(ops, hd):
    """Powers of two that go from the queries to the keys change no bit, however small the queries get; small keys and values keep theirs."""
    q, k, v = rnd(150, 4, hd, seed=31), rnd(150, 2, hd, seed=32), rnd(150, 2, hd, seed=33)
    out = attend(ops, q, k, v)
    assert torch.equal(attend(ops, q * 2.0 ** -95, k * 2.0 ** 95, v), out)
    s = torch.einsum("thd,shd->hts", q.double(), k.double().repeat_interleave(2, 1)) * hd ** -0.5
    s = s.masked_fill(torch.ones(150, 150, dtype=torch.bool, device=DEV).triu(1), -math.inf)
    want = torch.einsum("hts,shd->thd", torch.softmax(s, -1), v.double().repeat_interleave(2, 1))
    # a score's error moves a weight by as much: hd + 8 roundings of the largest sum of products
    bound = (hd + 8) * 2.0 ** -23 * float(s.abs()[s > -math.inf].max() + 1) * float(v.abs().max())
    for power in (80, 95, 120):                            # (queries below and above 2^90)
        kk = k * 2.0 ** -power
        exact = (kk * 2.0 ** power).double()               # (what is left of keys below the smallest normal float)
        s2 = torch.einsum("thd,shd->hts", q.double(), exact.repeat_interleave(2, 1)) * hd ** -0.5
        want2 = torch.einsum("hts,shd->thd", torch.softmax(s2.masked_fill(s == -math.inf, -math.inf), -1), v.double().repeat_interleave(2, 1))
        assert (attend(ops, q * 2.0 ** power, kk, v).double() - want2).abs().max() <= bound, power
    small = attend(ops, q, k, v * 2.0 ** -100).double() * 2.0 ** 100
    assert (small - want).abs().max() <= bound
    top = attend(ops, q, k, v * 2.0 ** 100).double() * 2.0 ** -100
    assert (top - want).abs().max() <= bound


def plain_attention(q, k, v, slopes=None, softcap=0.0, window=0):
    """In 64 bits, with the largest |score|."""
    n, nh, hd = q.shape
    group = nh // k.shape[1]
    s = torch.einsum("thd,shd->hts", q.double(), k.double().repeat_interleave(group, 1)) * hd ** -0.5
    if softcap:
        s = softcap * torch.tanh(s / softcap)
    pos = torch.arange(n, device=DEV)
    away = (pos[:, None] - pos[None, :]).double()
    if slopes is not None:
        s = s - slopes.double()[:, None, None] * away
    hidden = (away < 0) | ((away >= window) if window else (away < 0))
    most = float(s.masked_fill(hidden, 0.0).abs().max())
    return torch.einsum("hts,shd->thd", torch.softmax(s.masked_fill(hidden, -math.inf), -1), v.double().repeat_interleave(group, 1)), most


@pytest.mark.parametrize("hd,vd", [(48, 48), (80, 112), (128, 128), (64, 16)])
@pytest.mark.parametrize("how", ["slopes", "softcap", "both", "window"])
def test_attention_options_over_a_portion(ops, hd, vd, how):
    """Slopes, bounds of scores and windows over several tiles and splits of a portion."""
    n, nh, nkv = 300, 6, 2
    q, k, v = rnd(n, nh, hd, seed=40), rnd(n, nkv, hd, seed=41), rnd(n, nkv, vd, seed=42)
    slopes = torch.tensor([2.0 ** -i for i in range(nh)], device=DEV) if how in ("slopes", "both") else None
    softcap, window = (3.0 if how in ("softcap", "both") else 0.0), (70 if how == "window" else 0)
    want, most = plain_attention(q, k, v, slopes, softcap, window)
    out = attend(ops, q, k, v, 128, window, slopes, softcap)
    # a score's error moves a weight by as much: hd + 8 roundings of the largest score (slopes reach n), and those of the row's sums
    assert (out.double() - want).abs().max() <= ((hd + 8) * (most + 1) + n) * 2.0 ** -24 * float(v.abs().max())


@pytest.mark.parametrize("hd", [48, 128])
@pytest.mark.parametrize("split", [64, 256])
def test_attention_of_keys_that_are_not_finite(ops, hd, split):
    """Infinite keys and ones that are no numbers, in both halves of tiles: rows that see one are what 64 bits make of them, others are
    untouched."""
    n, nh, nkv = 300, 4, 2
    q, k, v = rnd(n, nh, hd, seed=43), rnd(n, nkv, hd, seed=44), rnd(n, nkv, hd, seed=45)
    fine = attend(ops, q, k, v, split)
    k[40, 0, 3], k[100, 1, 0], k[170, 0, 5], k[255, 1, 1] = -math.inf, math.inf, math.nan, 1e37
    want, _ = plain_attention(q, k, v)
    out = attend(ops, q, k, v, split)
    assert torch.equal(out[:40], fine[:40]) and torch.equal(torch.isnan(out), torch.isnan(want))
    same = torch.isfinite(want)
    # (row 255 on: keys next to the largest float, whose scores decide alone)
    assert float(((out.double() - want).abs())[same].max()) <= (hd + 8) * 2.0 ** -20 * float(v.abs().max())
