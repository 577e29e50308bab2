"""Gates of results that leave as bfloat16, held to 64 bits from nearly shut to wide open: what they are multiplied with is good to float's last bits, so
that a result is its exact value rounded once, whichever kernel makes it."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def rounded_once(got, want, slack):
    """Whether bfloat16 `got` is `want` rounded to the nearest, from a value at most `slack` off."""
    half = torch.exp2(torch.floor(torch.log2(want.abs().clamp_min(2.0 ** -126))) - 8)      # half the last of 8 bits
    return bool(((got.double() - want).abs() <= half + slack).all())


@pytest.mark.parametrize("col", [8, 7])                    # rows in pieces of 16 bytes, and off them
@pytest.mark.parametrize("after", [False, True])
@pytest.mark.parametrize("src_dtype", [torch.float32, torch.bfloat16])
def test_norm_with_gates(col, after, src_dtype):
    from beglin_b200.csrc import ops
    T, inner, groups, eps = 48, 1024, 2, 1e-5
    g = torch.Generator().manual_seed(col)
    z = torch.empty(T, inner).uniform_(-88.5, 88.5, generator=g)
    z[:, ::5].uniform_(-88.5, -87.0, generator=g)          # where 1 + e^-z lies above 2^126
    z = z.to(src_dtype).clamp(-88.5, 88.5)
    y = torch.empty(T, inner).uniform_(0.5, 2.0, generator=g)
    w = torch.empty(inner).uniform_(0.5, 2.0, generator=g) * 2.0 ** 60
    src = torch.full((T, inner + 16), float("nan"), dtype=src_dtype)
    src[:, col:col + inner] = z
    out = torch.full((T, inner), float("nan"), dtype=torch.bfloat16, device=DEV)
    ops.gated_group_rmsnorm(y.to(DEV), src.to(DEV), col, w.to(DEV), eps, groups, out, gate_after=after)
    y, z, w = y.double(), z.double(), w.double()
    v = y if after else y * z * torch.sigmoid(z)
    inv = 1.0 / torch.sqrt(v.view(T, groups, -1).square().mean(-1) + eps).repeat_interleave(inner // groups, 1)
    want = v * inv * w * (torch.sigmoid(z) if after else 1.0)
    # twelve roundings of float (exponential, sum, quotient, norm, products); a gate below 2^-126 keeps 2^-150 of its own
    assert rounded_once(out.cpu(), want, 12 * 2.0 ** -24 * want.abs() + (y * inv * w).abs() * 2.0 ** -149)
