"""Float products whose inner size is cut into ranges: the ranges' sums in rows of whole 16-byte pieces (four outputs a thread) and off them (one)
give the same bits, with and without a bias and the values that were there, and nothing is written beside the outputs."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("M,N,K", [(1, 4, 600), (3, 100, 640), (70, 1536, 1536), (65, 132, 9000), (17, 131, 2048)])
@pytest.mark.parametrize("bias", [False, True])
@pytest.mark.parametrize("accumulate", [False, True])
def test_sums_of_ranges(M, N, K, bias, accumulate):
    from beglin_b200.csrc import ops
    g = torch.Generator().manual_seed(M + N + K)
    a, w, old, b = (torch.randn(*s, generator=g).to(DEV) for s in ((M, K), (N, K), (M, N), (N,)))
    got = []
    for pad, at in ((4, 0), (4, 4), (1, 0), (3, 1)):
        buf = torch.full((M, N + pad + at), 7.0, device=DEV)
        out = buf[:, at:at + N]
        out.copy_(old)
        ops.gemm_f32_nt(a, w, b if bias else None, out, accumulate=accumulate)
        got.append(out.clone())
        assert (buf[:, :at] == 7.0).all() and (buf[:, at + N:] == 7.0).all()
    assert all(torch.equal(got[0], o) for o in got[1:])
    want = a.double() @ w.double().T + (b.double() if bias else 0.0) + (old.double() if accumulate else 0.0)
    # every term and every sum of the K of them is rounded to 2^-24 of what it is at most
    bound = 2.0 ** -24 * K * (a.double().abs() @ w.double().abs().T) / 8 + 2.0 ** -22 * (1.0 + want.abs())
    assert ((got[0].double() - want).abs() <= bound).all()
