"""Complete products of few rows, whose ranges of the inner size are added inside a cluster, around the numbers of rows at which the
kernel's tiles and the number of ranges change."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("N,K", [(264, 72), (576, 1024), (2624, 4096), (6152, 520), (9216, 1536), (40, 4096)])
@pytest.mark.parametrize("T", [1, 16, 17, 32, 33, 64])
def test_complete_products_of_few_rows(N, K, T):
    from beglin_b200.csrc import ops
    from beglin_b200.parts import BuildContext
    from beglin_b200.parts.linear import Linear
    ctx = BuildContext(device=DEV, compute_dtype=torch.bfloat16)
    ctx.status = ops.new_status(DEV)
    g = torch.Generator().manual_seed(N + T)
    w, b, x = torch.randn(N, K, generator=g), torch.randn(N, generator=g), torch.randn(T, K, generator=g).to(DEV, torch.bfloat16)
    for bias in (None, b):
        lin = Linear(w, bias, ctx)
        exact, size = x.double() @ lin.weight.double().T, x.double().abs() @ lin.weight.double().abs().T
        if bias is not None:
            exact, size = exact + lin.bias_f32.double(), size + lin.bias_f32.double().abs()
        full, short = lin.full_f32(x), lin(x)
        ops.raise_on_status(ctx.status)
        assert full.dtype == torch.float32 and short.dtype == torch.bfloat16
        off = K * 2.0 ** -24 * size                           # sums of K products in float
        assert ((full.double() - exact).abs() <= off).all()
        assert ((short.double() - exact).abs() <= off + 2.0 ** -8 * (exact.abs() + off)).all()


def test_complete_product_of_no_rows():
    from beglin_b200.csrc import ops
    from beglin_b200.parts import BuildContext
    from beglin_b200.parts.linear import Linear
    ctx = BuildContext(device=DEV, compute_dtype=torch.bfloat16)
    ctx.status = ops.new_status(DEV)
    lin = Linear(torch.randn(264, 72), None, ctx)
    out = lin(torch.empty(0, 72, dtype=torch.bfloat16, device=DEV))
    assert out.shape == (0, 264) and out.dtype == torch.bfloat16


def test_short_inner_sizes_are_not_cut():
    from beglin_b200.parts import BuildContext
    from beglin_b200.parts.tensor_core import TensorCoreProduct
    for k, cut in ((72, False), (520, False), (960, False), (1024, True), (4096, True)):
        p = TensorCoreProduct(torch.empty((576, k), dtype=torch.bfloat16, device=DEV), BuildContext(device=DEV, compute_dtype=torch.bfloat16))
        assert all((p.complete_splits(T) > 1) == cut for T in (1, 16, 33, 64)), k
