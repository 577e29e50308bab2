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


@pytest.mark.parametrize("col", [4, 3])                    # two channels a thread, and one
@pytest.mark.parametrize("chunked", [False, True])
def test_recurrence_with_its_branch(col, chunked):
    from beglin_b200.csrc import ops
    from beglin_b200.engine.batch import cut_long_requests
    T, W = 70, 512
    g = torch.Generator().manual_seed(col)
    z = torch.empty(T, W).uniform_(-10.06, 12.0, generator=g)
    z[:, ::4].uniform_(-10.06, -9.98, generator=g)          # where 1 + e^x lies above 2^126
    z[:, 1::4].uniform_(-2.0, 2.0, generator=g)
    z[0, :4] = torch.tensor([90.0, -90.0, 1e20, -1e20])
    src = torch.full((T, W + 8), float("nan"), device=DEV)
    src[:, col:col + W] = z.to(DEV)
    zero, S = torch.zeros(W, device=DEV), torch.empty(1, W).uniform_(0.5, 2.0, generator=g) * 2.0 ** 40
    state, slots = S.to(DEV), torch.zeros(1, dtype=torch.int32, device=DEV)            # no decay, no input: the state stays
    args = (torch.zeros(1, T, 2 * W, device=DEV), torch.zeros(T, W, device=DEV), src, col, zero, zero, zero, state, slots)
    out = torch.full((T, W), float("nan"), dtype=torch.bfloat16, device=DEV)
    if chunked:
        _, chunks, longs = cut_long_requests([0], [T], 32, 1)
        ops.rglru_scan(*args, None, 0, out, chunked=(torch.from_numpy(chunks).to(DEV), chunks.shape[0], torch.from_numpy(longs).to(DEV), longs.shape[0], 32))
    else:
        ops.rglru_scan(*args, torch.tensor([[0, 0, T]], dtype=torch.int32, device=DEV), 1, out)
    z, S = z.double(), S.double()
    x = 2.0 * 0.7978845608028654 * (z + 0.044715 * z ** 3)
    want = S * z * torch.sigmoid(x)
    # eight roundings of float; those of x (five, three of them in z^3) move a shut gate by x times themselves; from e^88.7 on it is nought
    off = (8 + 6 * x.abs().clamp_max(90.0) * (x < 0)) * 2.0 ** -24 * want.abs() + S * z.abs() * 2.0 ** -127.9 * (x < 0)
    assert rounded_once(out.cpu(), want, off) and torch.equal(state.cpu().double(), S)
