"""Chunked linear attention whose decays come from a short row through a matrix: ranks on both sides of what is staged at once, of whole
16-byte pieces and not, heads that take 8, 16 and 32 lanes a key, against the recurrence token by token."""
import pytest
import torch

from dinatar_helpers import rel_err
from test_dinatar_parts import DEV, Linear, NAN, ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,rank,pad", [(24, 4, 4), (32, 16, 4), (36, 3, 4), (64, 8, 4), (100, 16, 4), (128, 16, 3), (128, 20, 4), (132, 12, 4), (256, 40, 4)])
def test_decays_of_any_rank(n, rank, pad):
    from beglin_b200.engine.batch import cut_long_requests
    H, nv, lens = 2, 24, [130, 63, 17]
    L = Linear(False, H, n, nv, seed=n + rank, rank=rank)
    shift = pad - L.pad
    L.pad, L.cols, L.width = pad, {c: at + shift for c, at in L.cols.items()}, (L.width + shift + 3) // 4 * 4
    starts = [0, 130, 193]
    assert ops().gla_chunk(n, nv)
    rows = L.rows(sum(lens))
    state = torch.zeros(3, H * n * nv, device=DEV)
    _, chunks, longs = cut_long_requests(starts, lens, ops().gla_chunk(n, nv), 16)
    up = lambda a: torch.from_numpy(a).to(DEV)
    out = torch.full((sum(lens), H * nv), NAN, device=DEV)
    L.run(rows, state, torch.arange(3, dtype=torch.int32, device=DEV), out, chunks=up(chunks), longs=up(longs))
    for i in range(3):
        sl = slice(starts[i], starts[i] + lens[i])
        want, S = L.want(rows[sl], None)
        assert rel_err(out[sl], want) < 2e-5, i                      # (the bounds of the part's other tests, sums of the same length)
        assert rel_err(state[i].view(H, n, nv), S) < 5e-6, i
