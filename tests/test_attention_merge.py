"""The merge of a few ranges of keys: four features a lane (rows of whole 16-byte pieces) against the one-feature form (rows off them), which must
give the same bits, and both against 64 bits; parts of ranges that a row does not see hold NaN."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("hd", [4, 32, 64, 100, 128])
@pytest.mark.parametrize("T,H,splits,split", [(1, 1, 1, 64), (5, 3, 8, 64), (150, 5, 7, 0), (3, 2, 16, 32), (70, 12, 9, 0)])
@pytest.mark.parametrize("window,keep,sink", [(0, 0, 0), (200, 0, 1), (150, 40, 0)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_merge_of_a_few_ranges(hd, T, H, splits, split, window, keep, sink, dtype):
    from beglin_b200.csrc import ops
    g = torch.Generator().manual_seed(hd + T + splits)
    longest = splits * (split or 256)
    pos = torch.randint(0, longest, (T,), generator=g)
    pos[0] = longest - 1
    o, m, l = torch.randn(T, H, splits, hd, generator=g), 4 * torch.randn(T, H, splits, generator=g), 0.5 + torch.rand(T, H, splits, generator=g)
    sinks = torch.randn(H, generator=g)
    want = torch.zeros(T, H, hd, dtype=torch.float64)
    for t in range(T):
        p = int(pos[t])
        per = split or max(256, -(-(-(-(p + 1) // splits)) // 256) * 256)
        lo = max(0, p - window + 1) if window else 0
        for s in range(splits):
            if (s < lo // per and s > ((keep - 1) // per if keep else -1)) or s > p // per:
                o[t, :, s], m[t, :, s], l[t, :, s] = math.nan, math.nan, math.nan
        seen = ~m[t, 0].isnan()
        ms, ls, os = m[t][:, seen].double(), l[t][:, seen].double(), o[t][:, seen].double()
        top = ms.max(1).values
        if sink:
            top = torch.maximum(top, sinks.double())
        f = torch.exp(ms - top[:, None])
        den = (ls * f).sum(1) + (torch.exp(sinks.double() - top) if sink else 0.0)
        want[t] = (os * f[:, :, None]).sum(1) / den[:, None]
    dev = [x.to(DEV).contiguous() for x in (o, torch.stack([m, l], -1), pos.int())]
    sw = sinks.to(DEV)
    outs = []
    for stride in (H * hd, H * hd + 1):
        out = torch.full((T, stride), math.nan, device=DEV, dtype=dtype)
        ops._check(ops.lib().bg_attention_merge(ops._p(dev[0]), ops._p(dev[1]), ops._p(dev[2]), ops._p(out), ops._dt(out), stride, T, H, hd, splits, split,
                                                window, sink, ops._p(sw), keep, ops._stream()), "attention_merge")
        outs.append(out[:, :H * hd].cpu())
    if not (splits > 8 and T * H <= 128 and dtype == torch.bfloat16):            # (a kernel of its own takes those, whatever the stride)
        assert torch.equal(outs[0], outs[1])
    # a result is a sum of at most 16 terms whose weights' exponentials are good to 2 x 2^-23 and whose exponents are rounded (|m| < 32); it is up to
    # twice the largest part (the sums l are a half and more), and bfloat16 rounds it to 2^-8 of itself
    rel = 2 * ((16 + 32) * 2.0 ** -23 + (2.0 ** -8 if dtype == torch.bfloat16 else 0.0))
    scale = (o.nan_to_num().abs().amax(2)).double()
    for out in outs:
        assert ((out.view(T, H, hd).double() - want).abs() <= rel * scale + 1e-30).all()
