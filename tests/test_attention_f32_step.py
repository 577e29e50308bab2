"""Float attention of a step as one call beside its entries: the same bits in the addend and in the cache."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("how", [{}, {"qkv_bias": False, "out_bias": True}, {"window": 40}, {"window": 40, "keep_first": 3}, {"block": 32}, {"sink": True},
                                 {"sink": "learned"}, {"score_cap": 20.0}, {"head_dim": 64, "rot": 32}, {"head_dim": 20, "rot": 20}])
@pytest.mark.parametrize("lens,held", [([1], [3]), ([1, 1, 1], [600, 70, 64]), ([150, 3], [0, 300]), ([33, 1, 8], [5, 30, 0])])
def test_one_call_gives_the_bits_of_the_single_entries(how, lens, held):
    from beglin_b200.csrc import ops
    from beglin_b200.parts import AttentionSpec, BuildContext, PositionSpec
    from beglin_b200.parts.attention import GQAAttention
    from test_sukisun_parts import Requests
    how = dict(how)
    hd, rot = how.pop("head_dim", 128), how.pop("rot", None)
    spec = AttentionSpec(**{**dict(hidden=200, n_heads=6, n_kv_heads=2, head_dim=hd, qkv_bias=True, position=PositionSpec(rotary_dim=rot or hd, theta=1000.0)), **how})
    ctx = BuildContext(device=DEV, compute_dtype=torch.float32, page_size=64, status=ops.new_status(DEV))
    g = torch.Generator().manual_seed(hd + sum(lens))
    w = {r.name: torch.randn(r.shape, generator=g) * (r.shape[-1] ** -0.5 if len(r.shape) > 1 else 0.3) for r in GQAAttention.expected_tensors(spec)}
    part = GQAAttention(spec, w, ctx)
    assert part._args is not None
    outs, pools, launched = [], [], []
    for one in (True, False):
        if not one:
            part._args = None
        reqs = Requests([GQAAttention.cache_need(spec, ctx)], 64, torch.float32, pages=sum(-(-(n + h) // 64) + 1 for n, h in zip(lens, held)), slots=len(lens))
        pool = reqs.cache.kv_groups[0].device_pool
        pool.copy_(torch.randn(pool.shape, generator=torch.Generator().manual_seed(5)).to(DEV))
        if any(held):
            reqs.batch([(i, n) for i, n in enumerate(held) if n])
        b = reqs.batch([(i, n) for i, n in enumerate(lens)])
        h = torch.randn(sum(lens), 200, generator=torch.Generator().manual_seed(6)).to(DEV)
        part.position.table(b)                             # (made once a step)
        before = ops.launch_count()
        outs.append(part.forward(h, b, reqs.cache.view(0, b)))
        launched.append(ops.launch_count() - before)
        pools.append(pool.clone())
    assert torch.equal(outs[0], outs[1]) and torch.equal(pools[0], pools[1]) and launched[0] == launched[1] and not outs[0].isnan().any()
    ops.raise_on_status(ctx.status)
