"""The float feed-forward as one call beside its three entries: the same bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("T,hidden,ff,block", [(1, 64, 128, 64), (8, 256, 576, 64), (16, 200, 1028, 0), (17, 768, 2304, 64), (64, 136, 544, 4), (65, 132, 640, 64),
                                               (300, 256, 1600, 0), (550, 384, 8960, 64)])
@pytest.mark.parametrize("act", ["silu", "gelu_tanh", "glu_clamped"])
def test_one_call_gives_the_bits_of_three(T, hidden, ff, block, act):
    from beglin_b200.csrc import ops
    g = torch.Generator().manual_seed(T + ff)
    rnd = lambda *n: torch.randn(*n, generator=g).to(DEV)
    h, up, down, status = rnd(T, hidden + 4)[:, :hidden], rnd(2 * ff, hidden) * hidden ** -0.5, rnd(hidden, ff) * ff ** -0.5, ops.new_status(DEV)
    if T > 1:
        h[T // 2, 3] = float("inf")                        # a row whose sums floats make
    limit = 1.5 if act == "glu_clamped" else 0.0
    gu, rows, want = torch.empty(T, 2 * ff, device=DEV), torch.empty(T, ff, device=DEV), torch.empty(T, hidden, device=DEV)
    ops.gemm_f32_nt(h, up, None, gu, status=status)
    ops.swiglu(gu, rows, block, act, limit)
    ops.gemm_f32_nt(rows, down, None, want, status=status)
    got = ops.mlp_f32(h, up, block, down, act, limit, status)
    ops.raise_on_status(status)
    assert torch.equal(got.view(torch.int32), want.view(torch.int32))
