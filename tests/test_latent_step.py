"""Attention through a latent in steps of few rows: the per-head products against 64-bit sums at the edges of their tiles, and the step as one call beside
the same step entry by entry."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("H,T,K,N", [(1, 1, 64, 8), (3, 7, 64, 320), (2, 16, 128, 128), (20, 17, 448, 64), (5, 33, 704, 132), (32, 64, 512, 128), (40, 130, 64, 260)])
@pytest.mark.parametrize("form", ["columns", "heads"])
@pytest.mark.parametrize("gate", [None, "head", "feature"])
def test_per_head_products(H, T, K, N, form, gate):
    from beglin_b200.csrc import ops
    g = torch.Generator().manual_seed(H * T + K)
    rnd = lambda *n: torch.randn(*n, generator=g).to(DEV, torch.bfloat16)
    if form == "columns":                                  # a head's rows begin at a column of their own, other columns between
        x = rnd(T, H * (K + 24))
        x.view(T, H, K + 24)[:, :, K:] = float("nan")
        x = x.view(T, H, K + 24)[:, :, :K].transpose(0, 1)
    else:
        x = rnd(H, T, K)
    w, status = rnd(H, N, K), ops.new_status(DEV)
    want, size = x.double() @ w.double().transpose(1, 2), x.double().abs() @ w.double().abs().transpose(1, 2)
    off = K * 2.0 ** -24 * size                            # float sums of K products
    if gate is None:
        out = torch.full((H, T, N + 4), 7.0, device=DEV)[:, :, :N]
        ops.gemm_heads(x, w, out, status)
        assert ((out.double() - want).abs() <= off).all()
    else:
        gates = torch.randn(T, 3 + H * N, generator=g).to(DEV, torch.float32 if T % 2 else torch.bfloat16)
        out = torch.full((T, H * N), 7.0, dtype=torch.bfloat16, device=DEV)
        ops.gemm_heads(x, w, out, status, gates, 3, per_feature=gate == "feature")
        s = torch.sigmoid(gates[:, 3:].double())
        s = s.view(T, H, N) if gate == "feature" else s[:, :H, None]
        want, off = want.transpose(0, 1) * s, off.transpose(0, 1) * s
        assert ((out.view(T, H, N).double() - want).abs() <= off * (1 + 2.0 ** -8) + (2.0 ** -8 + 2.0 ** -20) * want.abs()).all()
    ops.raise_on_status(status)


@pytest.mark.parametrize("how", [{}, {"gated": False}, {"window": 70}, {"gate_features": True}, {"sink": True}, {"rot_dim": 32}])
@pytest.mark.parametrize("lens,held", [([1], [3]), ([1] * 5, [600, 70, 1, 130, 64]), ([1] * 40, [200 + i for i in range(40)]), ([20, 1], [5, 300]), ([64], [0]), ([65], [10])])
def test_one_call_gives_the_bits_of_the_single_entries(how, lens, held):
    from beglin_b200.csrc import ops
    from beglin_b200.parts import BuildContext, LatentAttentionSpec, PositionSpec
    from beglin_b200.parts.latent_attention import LatentAttention
    from test_sukisun_parts import Requests, latent_weights
    rot = how.get("rot_dim", 64)
    spec = LatentAttentionSpec(**{**dict(hidden=192, n_heads=6, dim=64, rot_dim=rot, vdim=72, q_rank=128, kv_rank=192, scale=0.1, eps=1e-5,
                                         position=PositionSpec(rotary_dim=rot, theta=1000.0, pairing="interleaved")), **how})
    ctx = BuildContext(device=DEV, compute_dtype=torch.bfloat16, page_size=64, status=ops.new_status(DEV))
    part = LatentAttention(spec, latent_weights(spec, 7, torch.bfloat16), ctx)
    assert part._args is not None
    outs, pools, launched = [], [], []
    for one in (True, False):
        reqs = Requests([LatentAttention.cache_need(spec)], 64, torch.bfloat16, pages=sum(-(-(n + h) // 64) for n, h in zip(lens, held)), slots=len(lens))
        reqs.cache.kv_groups[0].device_pool.copy_(torch.randn(reqs.cache.kv_groups[0].device_pool.shape, generator=torch.Generator().manual_seed(5)).to(DEV, torch.bfloat16))
        if any(held):
            reqs.batch([(i, n) for i, n in enumerate(held) if n])
        b = reqs.batch([(i, n) for i, n in enumerate(lens)])
        h = torch.randn(sum(lens), 192, generator=torch.Generator().manual_seed(6)).to(DEV, torch.bfloat16)
        if not one:
            part._args = None
        took = part._one_call(h, b, reqs.cache.view(0, b)) is not None
        assert took == (one and sum(lens) <= 64 and not (how.get("gate_features") and sum(lens) >= part.WIDE_ROWS))
        part.position.table(b)                             # (made once a step)
        before = ops.launch_count()
        outs.append(part.forward(h, b, reqs.cache.view(0, b)))
        launched.append(ops.launch_count() - before)
        pools.append(reqs.cache.kv_groups[0].device_pool.clone())
    assert torch.equal(outs[0], outs[1]) and torch.equal(pools[0], pools[1]) and launched[0] == launched[1]
    ops.raise_on_status(ctx.status)


@pytest.mark.parametrize("H,T,N", [(48, 49, 72), (48, 64, 72), (80, 64, 72), (80, 61, 8), (50, 64, 100), (80, 200, 132)])
@pytest.mark.parametrize("gate", [None, "head", "feature"])
def test_per_head_products_whose_features_end_inside_a_warp(H, T, N, gate):
    """More rows a CTA than one load of tensor memory gives (two loads of 16 columns and more), where lanes of a warp have no feature to store."""
    from beglin_b200.csrc import ops
    g = torch.Generator().manual_seed(H + T + N)
    rnd = lambda *n: torch.randn(*n, generator=g).to(DEV, torch.bfloat16)
    assert -(-N // 128) * H * -(-T // 16) > ops.sm_count() and N % 32
    x, w, status = rnd(H, T, 128), rnd(H, N, 128), ops.new_status(DEV)
    want, off = x.double() @ w.double().transpose(1, 2), 128 * 2.0 ** -24 * (x.double().abs() @ w.double().abs().transpose(1, 2))
    gates = None if gate is None else torch.randn(T, H * N, generator=g).to(DEV)
    out = torch.full((T, H * N + 4), 7.0, device=DEV)[:, :H * N]
    ops.gemm_heads(x, w, out, status, gates, 0, per_feature=gate == "feature")
    want, off = want.transpose(0, 1), off.transpose(0, 1)
    if gate is not None:
        s = torch.sigmoid(gates.double())
        s = s.view(T, H, N) if gate == "feature" else s[:, :H, None]
        want, off = want * s, off * s + 2.0 ** -20 * (want * s).abs()          # (the gate's own roundings)
    assert ((out.view(T, H, N).double() - want).abs() <= off).all()
    ops.raise_on_status(status)
