"""Routed experts in steps of many rows: the experts' products on pairs of CTAs over experts with no rows, a few and many, sizes that fill
no tile, and the kernels around them where their 16-byte forms begin and end."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def ops():
    from beglin_b200.csrc import ops as o
    o.lib()
    return o


CASES = [  # rows of the experts, rows behind them that no expert has, features in, features out
    ([129], 0, 64, 256), ([700, 0, 1], 0, 72, 264), ([0, 257, 256, 255, 128, 64], 5, 1000, 8), ([191, 192, 193, 385, 0, 600], 0, 512, 520),
    ([2048, 3], 0, 136, 1024), ([0, 0, 0, 900], 40, 328, 392), ([150] * 40, 0, 128, 128), ([1024] * 4, 0, 1536, 3072),
]


@pytest.mark.parametrize("rows,behind,K,N", CASES)
@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
def test_products_of_many_rows(ops, rows, behind, K, N, out_dtype):
    E, A = len(rows), sum(rows) + behind
    assert ops.grouped_pairs(A, E)
    g = torch.Generator().manual_seed(A + K)
    x = torch.randn(A, K, generator=g).to(DEV, torch.bfloat16)
    w = torch.randn(E, N, K, generator=g).to(DEV, torch.bfloat16)
    x[sum(rows):] = float("nan")
    starts = [sum(rows[:e]) for e in range(E + 1)]
    out, status = torch.full((A, N), 7.0, dtype=out_dtype, device=DEV), ops.new_status(DEV)
    ops.gemm_grouped(x, w, torch.tensor(starts, dtype=torch.int32, device=DEV), out, "relu2", status)
    ops.raise_on_status(status)
    for e in range(E):
        a, b = starts[e], starts[e + 1]
        z, size = x[a:b].double() @ w[e].double().T, x[a:b].double().abs() @ w[e].double().abs().T
        off = K * 2.0 ** -24 * size                           # sums of K float products
        want = z.clamp(min=0) ** 2
        bound = 2.0 * want.sqrt() * off + off * off + (2.0 ** -8 if out_dtype == torch.bfloat16 else 2.0 ** -23) * want
        assert ((out[a:b].double() - want).abs() <= bound).all(), (e, a, b)
    assert (out[sum(rows):] == 7.0).all()


@pytest.mark.parametrize("T,d", [(1, 8), (5, 24), (9, 36), (3, 7), (130, 1032), (33, 2048)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("scale", [False, True])
def test_rows_out_and_back(ops, T, d, dtype, scale):
    top, A = 3, 3 * T
    g = torch.Generator().manual_seed(T * d)
    x, y = torch.randn(T, d, generator=g).to(DEV, dtype), torch.randn(A, d, generator=g).to(DEV)
    weights, src_of = torch.rand(A, generator=g).to(DEV), torch.randperm(A, generator=g).to(DEV, torch.int32)
    row_of = torch.empty_like(src_of)
    row_of[src_of.long()] = torch.arange(A, dtype=torch.int32, device=DEV)
    xp, out = torch.full((A, d), float("nan"), dtype=dtype, device=DEV), torch.full((T, d), float("nan"), device=DEV)
    ops.route_gather(x, weights, src_of, xp, top, scale=scale)
    want = x[src_of.long() // top]
    assert torch.equal(xp, (weights[src_of.long()][:, None] * want.float()).to(dtype) if scale else want)
    ops.route_combine(y, weights, row_of, out, top, scale=scale)
    terms = y[row_of.long()].view(T, top, d).double() * (weights.view(T, top, 1).double() if scale else 1.0)
    assert ((out.double() - terms.sum(1)).abs() <= top * 2.0 ** -23 * terms.abs().sum(1)).all()


@pytest.mark.parametrize("T,E,top,d", [(1, 1, 1, 8), (8, 10, 2, 1536), (5, 16, 3, 264), (8, 8, 8, 64), (8, 40, 32, 512), (3, 130, 5, 2056), (7, 17, 17, 128)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_routing_of_few_tokens_in_one_kernel(ops, T, E, top, d, dtype):
    """The three kernels of a larger step as one: the same choices and weights bit for bit, a layout in which every expert holds its
    assignments, the same rows."""
    g = torch.Generator().manual_seed(T * E)
    h, W = torch.randn(T, d, generator=g).to(DEV, dtype), torch.randn(E, d, generator=g).to(DEV)
    bias, A = torch.randn(E, generator=g).to(DEV), T * top
    i32 = lambda *n: torch.full(n, -7, dtype=torch.int32, device=DEV)
    for scale_input in (False, True):
        for how in (dict(sigmoid="sigmoid", renorm=True), dict(sigmoid="softmax", bias=bias, scale=2.5), dict(sigmoid="softmax_chosen", logit_bias=bias)):
            ids, weights, offsets, row_of, src_of = i32(T, top), torch.zeros((T, top), device=DEV), i32(E + 1), i32(A), i32(A)
            xp = torch.full((A, d), float("nan"), dtype=dtype, device=DEV)
            assert ops.route_rows(h, W, top, ids, weights, offsets, row_of, src_of, xp, scale_input, **how)
            ids2, weights2, xp2 = i32(T, top), torch.zeros((T, top), device=DEV), torch.full_like(xp, float("nan"))
            ops.route(h, W, top, ids2, weights2, **how)
            assert torch.equal(ids, ids2) and torch.equal(weights, weights2)
            chosen, starts = ids.view(-1).long(), offsets.long()
            assert torch.equal(starts, torch.cat([torch.zeros(1, device=DEV), torch.bincount(chosen, minlength=E).cumsum(0)]).long())
            assert torch.equal(row_of[src_of.long()].long(), torch.arange(A, device=DEV))
            assert ((row_of.long() >= starts[chosen]) & (row_of.long() < starts[chosen + 1])).all()
            ops.route_gather(h, weights.view(-1), src_of, xp2, top, scale=scale_input)
            assert torch.equal(xp, xp2)


@pytest.mark.parametrize("T,E,top,d", [(9, 10, 2, 1536), (40, 8, 8, 64), (33, 200, 5, 2056), (256, 17, 3, 264), (257, 8, 2, 1536), (300, 40, 32, 72), (261, 120, 2, 136),
                                       (1003, 4, 2, 64), (700, 3, 3, 8), (2048, 16, 1, 1024), (2000, 9, 4, 520)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_routing_of_many_tokens_in_two_kernels(ops, T, E, top, d, dtype):
    """The same for steps of more tokens: edges of a warp's four tokens, of a block's, of a group of four experts, few columns and many."""
    g = torch.Generator().manual_seed(T * E)
    h, W = torch.randn(T, d, generator=g).to(DEV, dtype), torch.randn(E, d, generator=g).to(DEV)
    bias, A = torch.randn(E, generator=g).to(DEV), T * top
    i32 = lambda *n: torch.full(n, -7, dtype=torch.int32, device=DEV)
    for scale_input, how in ((False, dict(sigmoid="sigmoid", renorm=True)), (True, dict(sigmoid="softmax", bias=bias, scale=2.5))):
        ids, weights, offsets, row_of, src_of = i32(T, top), torch.zeros((T, top), device=DEV), i32(E + 1), i32(A), i32(A)
        xp = torch.full((A, d), float("nan"), dtype=dtype, device=DEV)
        assert ops.route_layout(h, W, top, ids, weights, offsets, row_of, src_of, xp, scale_input, i32(min(T * E, ops.ROUTE_LAYOUT_COUNTS)), **how)
        ids2, weights2, xp2, logits = i32(T, top), torch.zeros((T, top), device=DEV), torch.full_like(xp, float("nan")), torch.zeros((T, E), device=DEV)
        ops.route(h, W, top, ids2, weights2, logits=logits, **how)
        assert torch.equal(ids, ids2) and torch.equal(weights, weights2)
        assert ((logits.double() - h.double() @ W.double().T).abs() <= d * 2.0 ** -24 * (h.double().abs() @ W.double().abs().T)).all()
        chosen, starts = ids.view(-1).long(), offsets.long()
        assert torch.equal(starts, torch.cat([torch.zeros(1, device=DEV), torch.bincount(chosen, minlength=E).cumsum(0)]).long())
        assert torch.equal(src_of.long(), torch.sort(chosen, stable=True).indices)           # inside an expert: the order of the assignments
        assert torch.equal(row_of[src_of.long()].long(), torch.arange(A, device=DEV))
        ops.route_gather(h, weights.view(-1), src_of, xp2, top, scale=scale_input)
        assert torch.equal(xp, xp2)


def test_routing_of_many_tokens_refuses_what_it_does_not_take(ops):
    for T, E, d, n in ((2500, 256, 64, 8192), (300, 8, 36, 8192), (300, 8, 64, 100)):       # too many counts, rows of odd pieces, too little scratch
        h, W = torch.randn(T, d, device=DEV), torch.randn(E, d, device=DEV)
        i32 = lambda *n: torch.full(n, -7, dtype=torch.int32, device=DEV)
        ids = i32(T, 2)
        assert not ops.route_layout(h, W, 2, ids, torch.zeros((T, 2), device=DEV), i32(E + 1), i32(2 * T), i32(2 * T), torch.empty((2 * T, d), device=DEV),
                                    False, i32(n))
        assert (ids == -7).all()


@pytest.mark.parametrize("T,E,top,d,kernels", [(8, 10, 2, 64, 1), (9, 10, 2, 64, 3), (64, 40, 3, 1024, 2), (200, 40, 3, 1024, 3), (300, 40, 3, 1024, 2), (2000, 40, 3, 1024, 3),
                                               (5, 9, 2, 36, 3), (40, 300, 2, 1024, 3), (3, 1100, 2, 64, 3)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_routing_from_one_call(ops, T, E, top, d, kernels, dtype):
    """One, two or three kernels, whichever take the step: the same choices and weights, a layout in which every expert holds its rows, those rows."""
    g = torch.Generator().manual_seed(T + E)
    h, W = torch.randn(T, d, generator=g).to(DEV, dtype), torch.randn(E, d, generator=g).to(DEV)
    i32 = lambda *n: torch.full(n, -7, dtype=torch.int32, device=DEV)
    A = T * top
    ids, weights, offsets, row_of, src_of = i32(T, top), torch.zeros((T, top), device=DEV), i32(E + 1), i32(A), i32(A)
    xp = torch.full((A, d), float("nan"), dtype=dtype, device=DEV)
    before = ops.launch_count()
    assert ops.route_place(h, W, top, ids, weights, offsets, row_of, src_of, xp, True, i32(ops.route_layout_wins(T, d, E, top)), sigmoid="sigmoid")
    assert ops.launch_count() - before == kernels
    ids2, weights2, xp2 = i32(T, top), torch.zeros((T, top), device=DEV), torch.full_like(xp, float("nan"))
    ops.route(h, W, top, ids2, weights2, sigmoid="sigmoid")
    assert torch.equal(ids, ids2) and torch.equal(weights, weights2)
    chosen = ids.view(-1).long()
    assert torch.equal(offsets.long(), torch.cat([torch.zeros(1, device=DEV), torch.bincount(chosen, minlength=E).cumsum(0)]).long())
    assert torch.equal(torch.sort(src_of).values.long(), torch.arange(A, device=DEV)) and torch.equal(row_of[src_of.long()].long(), torch.arange(A, device=DEV))
    starts = offsets.long()
    assert ((row_of.long() >= starts[chosen]) & (row_of.long() < starts[chosen + 1])).all()
    ops.route_gather(h, weights.view(-1), src_of, xp2, top, scale=True)
    assert torch.equal(xp, xp2)
