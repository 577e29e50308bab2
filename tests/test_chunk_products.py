"""The recurrences' chunks on the tensor cores: float products from operands in three bfloat16 parts are held to the same bounds as the
float units' kernels, against the recurrence walked token by token in 64 bits."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def ops():
    from beglin_b200.csrc import ops as o
    o.lib()
    return o


def lists(lens, chunk):
    from beglin_b200.engine.batch import cut_long_requests
    starts = [sum(lens[:i]) for i in range(len(lens))]
    _, blocks, longs = cut_long_requests(starts, lens, chunk, 1)
    dev = lambda a: torch.tensor(a, dtype=torch.int32, device=DEV)
    return dev(blocks), len(blocks), dev(longs), len(longs)


def walk(a, k, v, q, S):
    """S <- diag(a_t) S + k_t v_t^T, o_t = S^T q_t over rows [n, heads, features]."""
    out = []
    for t in range(k.shape[0]):
        S = S * a[t][:, :, None] + k[t][:, :, None] * v[t][:, None, :]
        out.append((q[t][:, None, :] @ S)[:, 0])
    return torch.stack(out), S


def rnd(*shape, seed):
    g = torch.Generator().manual_seed(seed)
    return torch.randn(*shape, generator=g).to(DEV)


def close(got, want, terms):
    """Within `terms` roundings of 2^-24 of the largest value: a chunk's sums of some 200 products and the chunks' states."""
    assert float((got.double() - want).abs().max()) <= terms * 2.0 ** -24 * float(want.abs().max())


def walked_requests(make, lens, state0):
    """(outputs [T, ...], states) of every request by `walk`; `make(first row, rows)` gives (a, k, v, q)."""
    outs, states, row = [], [], 0
    for i, n in enumerate(lens):
        o, S = walk(*make(row, n), state0[i])
        outs.append(o.reshape(n, -1))
        states.append(S)
        row += n
    return torch.cat(outs), torch.stack(states)


SIZES = [(2, 128, 128, [64]), (3, 64, 48, [1, 65, 200]), (2, 96, 64, [130, 63]), (1, 64, 112, [700]), (2, 48, 128, [129]), (2, 48, 48, [64, 7]), (2, 32, 64, [70]),
         (1, 128, 144, [70])]


@pytest.mark.parametrize("H,n,nv,lens", SIZES)          # (the last two: sizes that stay with the float units)
def test_constant_decay(ops, H, n, nv, lens):
    T = sum(lens)
    src, decay = rnd(T, H * (2 * n + 2 * nv), seed=1), torch.tensor([0.0, 1.0 - 2.0 ** -8, 0.875][:H], device=DEV)
    state0 = rnd(len(lens), H, n, nv, seed=2)
    silu = lambda x: x * torch.sigmoid(x)

    def make(row, rows):
        x = silu(src[row:row + rows].double())
        q, k, v = x[:, :H * n].view(rows, H, n), x[:, H * n:2 * H * n].view(rows, H, n), x[:, 2 * H * n:2 * H * n + H * nv].view(rows, H, nv)
        return decay.double()[None, :, None].expand(rows, H, 1), k, v, q

    want, states = walked_requests(make, lens, state0.double())
    slots = torch.arange(len(lens) - 1, -1, -1, dtype=torch.int32, device=DEV)
    state = state0.flip(0).reshape(len(lens), -1).contiguous()
    y, status = torch.full((T, H * nv), float("nan"), device=DEV), ops.new_status(DEV)
    chunks, n_chunks, longs, n_long = lists(lens, ops.decay_attention_chunk(n, nv))
    ops.decay_attention(src, 0, H * n, 2 * H * n, decay, state, slots, None, 0, y, H, n, nv, chunks, n_chunks, longs, n_long, tensor_cores=True,
                        status=status)
    ops.raise_on_status(status)
    close(y, want, 64)
    close(state.flip(0).view_as(states), states, 64)


@pytest.mark.parametrize("H,n,nv,lens", SIZES)
@pytest.mark.parametrize("forget", [True, False])
def test_decay_per_channel(ops, H, n, nv, lens, forget):
    T, rank, qd, vd = sum(lens), 5, H * n, H * nv
    src = rnd(T, 2 * qd + 2 * vd + 8, seed=1)
    bias, lower, wa, norm_w = rnd(qd, seed=2), torch.rand(qd, generator=torch.Generator().manual_seed(3)).to(DEV), rnd(qd, rank, seed=4), rnd(nv, seed=5)
    state0 = rnd(len(lens), H, n, nv, seed=6)

    def make(row, rows):
        x = src[row:row + rows].double()
        q, f, v = x[:, :qd], x[:, qd:2 * qd], x[:, 2 * qd:2 * qd + vd].view(rows, H, nv)
        if forget:
            a = lower.double() + (1 - lower.double()) * torch.sigmoid(f + bias.double())
            k = 1 - a
        else:
            a, k = torch.sigmoid(x[:, 2 * qd + 2 * vd:2 * qd + 2 * vd + rank] @ wa.double().T + bias.double()) ** (1 / 16), f
        return a.view(rows, H, n), k.reshape(rows, H, n), v, q.reshape(rows, H, n) * 0.5

    want, states = walked_requests(make, lens, state0.double())
    want = want.view(T, H, nv)
    want = (want / ((want * want).mean(-1, keepdim=True) + 1e-6).sqrt() * norm_w.double()).reshape(T, -1)
    gate = src[:, 2 * qd + vd:2 * qd + 2 * vd].double()
    want = want * gate * torch.sigmoid(gate)
    slots = torch.arange(len(lens), dtype=torch.int32, device=DEV)
    state, status = state0.reshape(len(lens), -1).clone(), ops.new_status(DEV)
    out = torch.full((T, vd), float("nan"), dtype=torch.bfloat16, device=DEV)
    chunks, n_chunks, longs, n_long = lists(lens, ops.gla_chunk(n, nv))
    how = dict(lower=lower) if forget else dict(decay_matrix=wa, r_col=2 * qd + 2 * vd, power=1 / 16)
    ops.gated_linear_attention(src, 0, qd, 2 * qd, bias, norm_w, 1e-6, state, slots, None, 0, out, H, n, nv, q_scale=0.5, g_col=2 * qd + vd,
                               chunks=chunks, n_chunks=n_chunks, longs=longs, n_long=n_long, status=status, **how)
    ops.raise_on_status(status)
    close(state.view_as(states), states, 128)
    # (bfloat16 rounds a value to 2^-9 of it; the norm magnifies a head's own rounding where its values nearly cancel)
    assert float((out.double() - want).abs().max()) <= (2.0 ** -8 + 1e-4) * float(want.abs().max())


@pytest.mark.parametrize("H,P,N,G,lens", [(2, 128, 128, 1, [64]), (4, 80, 96, 2, [1, 65, 200]), (3, 96, 128, 1, [130, 63]), (2, 128, 112, 2, [700]), (2, 64, 128, 1, [70])])
def test_mamba2(ops, H, P, N, G, lens):
    T = sum(lens)
    xbc, raw = rnd(T, H * P + 2 * G * N, seed=1), rnd(T, H + 1, seed=2)
    bias, A_log, D = rnd(H, seed=3) - 1.0, rnd(H, seed=4), rnd(H, seed=5)
    raw[::9] += 6.0                                     # large steps that forget everything between small ones
    state0 = rnd(len(lens), H, N, P, seed=6)

    def make(row, rows):
        x = xbc[row:row + rows].double()
        B = x[:, H * P:H * P + G * N].view(rows, G, N).repeat_interleave(H // G, 1)
        C = x[:, H * P + G * N:].view(rows, G, N).repeat_interleave(H // G, 1)
        dt = torch.nn.functional.softplus(raw[row:row + rows, 1:].double() + bias.double())
        return torch.exp(-torch.exp(A_log.double()) * dt)[:, :, None], B, x[:, :H * P].view(rows, H, P) * dt[:, :, None], C

    want, states = walked_requests(make, lens, state0.double())
    want = want + (D.double()[:, None] * xbc[:, :H * P].double().view(T, H, P)).reshape(T, -1)
    slots = torch.arange(len(lens), dtype=torch.int32, device=DEV)
    state = state0.transpose(2, 3).reshape(len(lens), -1).contiguous()                      # a slot holds [H, P, N]
    y, status = torch.full((T, H * P), float("nan"), device=DEV), ops.new_status(DEV)
    chunks, n_chunks, longs, n_long = lists(lens, ops.ssm_chunk(H, P, N, G))
    ops.ssm_scan(xbc, raw, 1, bias, A_log, D, state, slots, None, 0, y, H, P, N, G, chunks, n_chunks, longs, n_long, tensor_cores=True, status=status)
    ops.raise_on_status(status)
    close(y, want, 64)
    close(state.view(len(lens), H, P, N).transpose(2, 3), states, 64)


def _decay(ops, bad):
    H, n, nv, T, at = 2, 64, 96, 150, 90
    src = rnd(T, H * (2 * n + 2 * nv), seed=1)
    src[at, 2 * H * n + nv + 5] = bad                    # head 1, value 5
    state, y = rnd(1, H * n * nv, seed=2), torch.full((T, H * nv), float("nan"), device=DEV)
    chunks, n_chunks, longs, n_long = lists([T], ops.decay_attention_chunk(n, nv))
    status = ops.new_status(DEV)
    ops.decay_attention(src, 0, H * n, 2 * H * n, torch.tensor([0.5, 0.875], device=DEV), state, torch.zeros(1, dtype=torch.int32, device=DEV), None, 0,
                        y, H, n, nv, chunks, n_chunks, longs, n_long, tensor_cores=True, status=status)
    ops.raise_on_status(status)
    return y.view(T, H, nv), state.view(H, n, nv), at


def _per_channel(ops, bad):
    H, n, nv, T, at = 2, 96, 64, 150, 90
    qd, vd = H * n, H * nv
    src = rnd(T, 2 * qd + 2 * vd, seed=1)
    src[at, 2 * qd + nv + 5] = bad
    state, out = rnd(1, H * n * nv, seed=6), torch.full((T, vd), float("nan"), dtype=torch.bfloat16, device=DEV)
    chunks, n_chunks, longs, n_long = lists([T], ops.gla_chunk(n, nv))
    status = ops.new_status(DEV)
    ops.gated_linear_attention(src, 0, qd, 2 * qd, rnd(qd, seed=2), rnd(nv, seed=5), 1e-6, state, torch.zeros(1, dtype=torch.int32, device=DEV), None, 0,
                               out, H, n, nv, lower=torch.full((qd,), 0.5, device=DEV), q_scale=0.5, g_col=2 * qd + vd, chunks=chunks,
                               n_chunks=n_chunks, longs=longs, n_long=n_long, status=status)
    ops.raise_on_status(status)
    return out.view(T, H, nv), state.view(H, n, nv), at


def _mamba2(ops, bad):
    H, P, N, T, at = 2, 80, 96, 150, 90
    xbc = rnd(T, H * P + 2 * N, seed=1)
    xbc[at, P + 5] = bad
    state, y = rnd(1, H * N * P, seed=6), torch.full((T, H * P), float("nan"), device=DEV)
    chunks, n_chunks, longs, n_long = lists([T], ops.ssm_chunk(H, P, N, 1))
    status = ops.new_status(DEV)
    ops.ssm_scan(xbc, rnd(T, H + 1, seed=2), 1, rnd(H, seed=3), rnd(H, seed=4), rnd(H, seed=5), state, torch.zeros(1, dtype=torch.int32, device=DEV), None, 0,
                 y, H, P, N, 1, chunks, n_chunks, longs, n_long, tensor_cores=True, status=status)
    ops.raise_on_status(status)
    return y.view(T, H, P), state.view(H, P, N).transpose(1, 2), at


@pytest.mark.parametrize("bad", [math.inf, math.nan, -3.4e38])
@pytest.mark.parametrize("run", [_decay, _per_channel, _mamba2], ids=["constant", "per_channel", "mamba2"])
def test_a_value_reaches_its_own_token_and_those_behind_it(ops, run, bad):
    """A value that is infinite, not a number or at float's end: the tokens of its chunk in front of it and the other heads keep their bits, and
    without a norm over the head the other features, too; its own column of the state holds it."""
    clean, clean_state, at = run(ops, 0.25)
    y, state, _ = run(ops, bad)
    assert torch.isfinite(clean).all() and torch.equal(y[:at], clean[:at]) and torch.equal(y[:, 0], clean[:, 0])
    assert torch.equal(state[0], clean_state[0])
    other = torch.arange(clean.shape[2], device=DEV) != 5
    assert torch.equal(state[1][:, other], clean_state[1][:, other])
    if run is not _per_channel:
        assert torch.equal(y[:, 1][:, other], clean[:, 1][:, other])
    if bad != -3.4e38:
        assert not torch.isfinite(y[at, 1, 5]) and not torch.isfinite(state[1][:, 5]).any()
