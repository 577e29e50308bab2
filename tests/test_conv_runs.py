"""The causal convolution in runs of rows: requests that begin anywhere in a run, shorter than the taps, beside runs that end early, with the state read
and written by the requests' own blocks, and the result's two bfloat16 numbers; against the same convolution a row at a time in 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("taps", [2, 3, 4])
@pytest.mark.parametrize("lens", [[96], [97, 1], [1, 2, 3, 100], [40, 8, 7, 65], [131, 9, 1, 1, 30]])
@pytest.mark.parametrize("w_dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("bias", [False, True])
def test_runs(taps, lens, w_dtype, bias):
    from beglin_b200.csrc import ops
    C, T, R, keep, blocks = 520, sum(lens), len(lens), taps - 1, 2
    assert ops.lib().bg_conv_silu_run(T, R) > 1
    g = torch.Generator().manual_seed(T * taps)
    rnd = lambda *n: torch.randn(*n, generator=g)
    src, w, b, sb, state = rnd(T, C + 12), rnd(C, taps).to(w_dtype), rnd(C).to(w_dtype), rnd(C) if bias else None, rnd(R + 1, 8 + keep * C)
    slots = torch.randperm(R + 1, generator=g)[:R].to(torch.int32)
    starts = [sum(lens[:i]) for i in range(R)]
    reqs = torch.tensor([[i, s, n] for i, (s, n) in enumerate(zip(starts, lens))], dtype=torch.int32)
    row_req = torch.cat([torch.full((n,), i, dtype=torch.int32) for i, n in enumerate(lens)])
    want, size, state2 = torch.zeros(T, C, dtype=torch.float64), torch.zeros(T, C, dtype=torch.float64), state.clone()
    for i, (s, n) in enumerate(zip(starts, lens)):
        old = state[slots[i]][8:].view(keep, C)
        new = src[s:s + n, 4:4 + C] + sb if bias else src[s:s + n, 4:4 + C]          # (rounded as the inputs are)
        seen = torch.cat([old, new])
        for k in range(taps):
            want[s:s + n] += w[:, k].double() * seen[k:k + n].double()
            size[s:s + n] += (w[:, k].double() * seen[k:k + n].double()).abs()
        state2[slots[i]][8:] = seen[n:].reshape(-1)
    want, size = want + b.double(), size + b.double().abs()
    to = lambda t: None if t is None else t.to(DEV)
    st, out, x2 = state.to(DEV), torch.full((T, C), float("nan"), device=DEV), torch.full((blocks, T, 2 * C // blocks), float("nan"), dtype=torch.bfloat16, device=DEV)
    before = ops.launch_count()
    ops.conv_silu(to(src), 4, C, to(w), to(b), st, 8, to(slots), to(row_req), to(reqs), R, out, activation="none", src_bias=to(sb), split=x2)
    assert ops.launch_count() - before == 1
    assert ((out.cpu().double() - want).abs() <= (taps + 1) * 2.0 ** -24 * size).all() and torch.equal(st.cpu(), state2)
    ref = torch.empty_like(x2)
    ops.rglru_split(out, blocks, ref)
    assert torch.equal(x2, ref)
    st2, silu = state.to(DEV), torch.full((T, C), float("nan"), device=DEV)
    ops.conv_silu(to(src), 4, C, to(w), to(b), st2, 8, to(slots), to(row_req), to(reqs), R, silu, src_bias=to(sb))
    z = out.double()
    assert ((silu.double() - z * torch.sigmoid(z)).abs() <= 2.0 ** -21 * (z * torch.sigmoid(z)).abs() + 2.0 ** -126).all() and torch.equal(st, st2)


@pytest.mark.parametrize("lens,C,blocks", [([1], 520, 2), ([5, 3], 520, 2), ([95], 520, 2), ([40] * 13, 520, 2), ([100], 516, 3), ([97], 35, 5), ([2] * 60, 64, 1)])
def test_split_of_steps_that_are_not_taken_in_runs(lens, C, blocks):
    """Few rows, many short requests, and sizes off 16 bytes: the convolution, its state and the split as kernels of their own, from the same call."""
    from beglin_b200.csrc import ops
    T, R, taps = sum(lens), len(lens), 4
    g = torch.Generator().manual_seed(T)
    rnd = lambda *n: torch.randn(*n, generator=g).to(DEV)
    src, w, b, state = rnd(T, C + 12), rnd(C, taps), rnd(C), rnd(R, 3 * C)
    starts = [sum(lens[:i]) for i in range(R)]
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    reqs, slots, row_req = i32([[i, s, n] for i, (s, n) in enumerate(zip(starts, lens))]), i32(list(range(R))), i32([i for i, n in enumerate(lens) for _ in range(n)])
    outs = []
    for split in (torch.full((blocks, T, 2 * C // blocks), float("nan"), dtype=torch.bfloat16, device=DEV), None):
        st, out = state.clone(), torch.full((T, C), float("nan"), device=DEV)
        before = ops.launch_count()
        ops.conv_silu(src, 4, C, w, b, st, 0, slots, row_req, reqs, R, out, activation="none", split=split)
        counted = ops.launch_count() - before
        if split is None:
            split = torch.empty_like(outs[0][2])
            ops.rglru_split(out, blocks, split)
            counted += 1
        outs.append((out, st, split, counted))
    assert all(torch.equal(x, y) for x, y in zip(outs[0][:3], outs[1][:3])) and outs[0][3] == outs[1][3] - (ops.lib().bg_conv_silu_run(T, R) > 1 and C % 4 == 0 and C // blocks % 4 == 0)
