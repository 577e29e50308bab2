"""Mamba-2 between its products as one call beside its entries: the same bits in the result and in the slots."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("heads,vdim,state,groups,conv", [(4, 16, 32, 2, 4), (3, 96, 96, 1, 4), (2, 20, 12, 1, 3)])
@pytest.mark.parametrize("steps", [[[1]], [[5, 1, 2]], [[300, 7], [1, 1]], [[64, 250, 3], [200, 0, 1]]])
def test_one_call_gives_the_bits_of_the_single_entries(dtype, heads, vdim, state, groups, conv, steps, monkeypatch):
    from beglin_b200.csrc import ops
    from beglin_b200.parts import BuildContext, Mamba2Spec
    from beglin_b200.parts.mamba2 import Mamba2
    from test_sukisun_parts import Requests
    spec = Mamba2Spec(hidden=72, n_heads=heads, vdim=vdim, state=state, groups=groups, conv=conv, norm_groups=1, eps=1e-5)
    ctx = BuildContext(device=DEV, compute_dtype=dtype, page_size=8, status=ops.new_status(DEV))
    g = torch.Generator().manual_seed(heads * vdim)
    w = {r.name: torch.randn(r.shape, generator=g) * (r.shape[-1] ** -0.5 if len(r.shape) > 1 else 0.5) for r in Mamba2.expected_tensors(spec)}
    part = Mamba2(spec, w, ctx)
    outs, slabs, launched = [], [], []
    for one in (True, False):
        reqs = Requests([Mamba2.cache_need(spec)], 8, dtype, pages=80, slots=max(len(s) for s in steps))
        reqs.cache.state_groups[0].slab.zero_()
        gen, got, n = torch.Generator().manual_seed(9), [], 0
        for lens in steps:
            b = reqs.batch([(i, k) for i, k in enumerate(lens) if k])
            h = torch.randn(sum(lens), 72, generator=gen).to(DEV, dtype)
            before = ops.launch_count()
            if one:
                got.append(part.forward(h, b, reqs.cache.view(0, b)))
            else:                                          # (entry by entry, as while kernel classes are timed)
                with monkeypatch.context() as m:
                    m.setattr(ops, "profiling", lambda: True)
                    got.append(part.forward(h, b, reqs.cache.view(0, b)))
            n += ops.launch_count() - before
        outs.append(torch.cat([o.float().sum(0) if o.dim() == 3 else o.float() for o in got]))
        slabs.append(reqs.cache.state_groups[0].slab.clone())
        launched.append(n)
    assert torch.equal(outs[0], outs[1]) and torch.equal(slabs[0], slabs[1]) and launched[0] == launched[1] and not outs[0].isnan().any()
    ops.raise_on_status(ctx.status)
