"""A step's routed experts as one call from the host beside the same step entry by entry: every form of layer, steps at the edges of what the
routing's kernels and the shared expert's products take."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def layer(form, experts, top, gen, hidden=192, ff=136, shared_ff=128):
    from beglin_b200.parts import registry
    from beglin_b200.parts.context import BuildContext
    from beglin_b200.parts.spec import RoutedExpertsSpec, SharedExpertSpec
    identity = 2 if form == "clamped" else 0
    how = {"plain": dict(activation="relu2"),
           "clamped": dict(activation="glu_clamped", limit=7.0, router_activation="softmax", choice_bias=True, route_scale=2.5, identity=identity,
                           scale_input=False, shared=SharedExpertSpec(intermediate=shared_ff, limit=5.0)),
           "silu": dict(activation="swiglu", router_activation="softmax_chosen", logit_bias=True, scale_input=False,
                        shared=SharedExpertSpec(intermediate=shared_ff, gated=False)),
           "silu_odd": dict(activation="swiglu", scale_input=False, shared=SharedExpertSpec(intermediate=40, gated=False))}[form]
    spec = RoutedExpertsSpec(hidden=hidden, intermediate=ff, experts=experts, top=top, **how)
    cls = registry.part_class("feed_forward", spec.kind)
    w = {r.name: torch.randn(r.shape, generator=gen).to(DEV, torch.bfloat16) * r.shape[-1] ** -0.5 for r in cls.expected_tensors(spec)}
    return cls(spec, w, BuildContext(device=DEV, compute_dtype=torch.bfloat16, page_size=64, status=torch.zeros(1, dtype=torch.int32, device=DEV)))


@pytest.mark.parametrize("form", ["plain", "clamped", "silu", "silu_odd"])
@pytest.mark.parametrize("T", [1, 8, 9, 16, 17, 65, 300, 1100])
def test_one_call_gives_the_bits_of_the_single_entries(form, T):
    gen = torch.Generator().manual_seed(T)
    part = layer(form, 4, 2, gen)
    h = torch.randn(T, 192, generator=gen).to(DEV, torch.bfloat16)
    from beglin_b200.csrc import ops
    assert part._args is not None
    before = ops.launch_count()
    got = part.forward(h, None)
    counted = ops.launch_count() - before
    part._args = None
    before = ops.launch_count()
    want = part.forward(h, None)
    assert torch.equal(got, want) and counted == ops.launch_count() - before
    ops.raise_on_status(part.ctx.status)


def test_one_call_leaves_sizes_of_odd_pieces_to_the_single_entries():
    gen = torch.Generator().manual_seed(0)
    assert layer("plain", 4, 2, gen, hidden=100)._args is None and layer("plain", 4, 2, gen, ff=36)._args is None
    part = layer("plain", 300, 2, gen)                      # more experts than the layout's counts take: the routing refuses, the step runs all the same
    h = torch.randn(40, 192, generator=gen).to(DEV, torch.bfloat16)
    assert part._one_call(h) is None and part.forward(h, None).shape == (40, 192)
    wide = torch.randn(8, 400, generator=gen).to(DEV, torch.bfloat16)
    assert layer("plain", 4, 2, gen)._one_call(wide[:, :192]) is None       # rows that do not lie one behind the other


@pytest.mark.parametrize("form,experts,T", [("clamped", 16, 2000), ("clamped", 62, 130), ("clamped", 62, 300), ("clamped", 62, 600), ("silu", 128, 65), ("silu", 64, 2048),
                                            ("clamped", 32, 250), ("silu_odd", 255, 40), ("silu", 300, 20), ("clamped", 1200, 3)])
def test_a_shared_expert_runs_once_whatever_the_routing_takes(form, experts, T):
    """Steps on both sides of what the routing's kernels take (300 outputs and more, and 8,192 counts), with a shared expert: the result and the launches of the
    single entries, and no result of the shared expert's that nobody uses."""
    from beglin_b200.csrc import ops
    gen = torch.Generator().manual_seed(T)
    part = layer(form, experts, 2, gen, hidden=64, ff=16)
    h = torch.randn(T, 64, generator=gen).to(DEV, torch.bfloat16)
    ran, shared = [], part._shared
    part._shared = lambda x: ran.append(x) or shared(x)
    before = ops.launch_count()
    got = part.forward(h, None)
    counted = ops.launch_count() - before
    once = len(ran)
    part._args = None
    before = ops.launch_count()
    want = part.forward(h, None)
    assert torch.equal(got, want) and counted == ops.launch_count() - before and once <= 1
    ops.raise_on_status(part.ctx.status)


def test_rows_off_16_bytes_run_the_shared_expert_once():
    from beglin_b200.csrc import ops
    gen = torch.Generator().manual_seed(0)
    part = layer("clamped", 4, 2, gen)
    rows = torch.randn(40 * 192, generator=gen).to(DEV, torch.bfloat16)
    off = torch.cat([rows.new_zeros(1), rows])[1:].view(40, 192)
    assert off.data_ptr() % 16
    ran, shared = [], part._shared
    part._shared = lambda x: ran.append(x) or shared(x.clone())      # (the products want their rows on 16 bytes)
    got = part.forward(off, None)
    assert len(ran) == 1
    want = part.forward(rows.view(40, 192), None)
    # (the router adds rows off 16 bytes up in another order: 192 x 2^-24 of logits below eight)
    assert float((got - want).norm() / want.norm()) < 1e-4
    ops.raise_on_status(part.ctx.status)


def test_scratch_of_the_layout_is_what_its_kernels_take():
    from beglin_b200.csrc import ops
    gen = torch.Generator().manual_seed(1)
    for T, E, top in [(9, 10, 2), (256, 32, 4), (257, 33, 1), (1820, 18, 2), (1824, 18, 2), (32, 256, 3), (33, 256, 3), (40, 257, 2), (2048, 8, 8)]:
        n = ops.route_layout_counts(T, 64, E, top)
        assert 0 <= n <= min(T * E, ops.ROUTE_LAYOUT_COUNTS)
        i32 = lambda k: torch.empty(k, dtype=torch.int32, device=DEV)
        args = (torch.randn(T, 64, generator=gen).to(DEV), torch.randn(E, 64, generator=gen).to(DEV), top, i32((T, top)), torch.zeros((T, top), device=DEV), i32(E + 1),
                i32(T * top), i32(T * top), torch.empty((T * top, 64), device=DEV), False)
        assert ops.route_layout(*args, i32(max(n, 1))) == (n > 0) and (n < 2 or not ops.route_layout(*args, i32(n - 1)))
    assert ops.route_layout_counts(64, 60, 8, 2) == 0


def test_scratch_holds_the_shared_experts_rows_only_where_they_are_made_in_the_call():
    from beglin_b200.csrc import ops
    part = layer("clamped", 4, 2, torch.Generator().manual_seed(1))
    up = lambda n: -(-n // 256) * 256
    for T in (8, 300):
        more = up(T * part.shared_up.out_features * 4) + up(T * 128 * 2) + up(T * 192 * 4)
        assert ops.experts_scratch(part._args, T, True) - ops.experts_scratch(part._args, T, False) == more
    for T in (8, 17, 300):
        part.forward(torch.randn(T, 192).to(DEV, torch.bfloat16), None)
        assert part._scratch[T] == ops.experts_scratch(part._args, T, part.shared_up.fuses(T))


@pytest.mark.parametrize("T,two", [(9, True), (128, True), (129, False), (256, False), (257, True), (1024, True), (1025, None)])
def test_routing_of_many_outputs_in_two_kernels_or_three(T, two):
    """32 outputs of 1,024 features, where the layout's kernel wins but for 129 to 256 tokens, up to its 8,192 counts."""
    from beglin_b200.csrc import ops
    gen = torch.Generator().manual_seed(T)
    part = layer("silu", 32, 2, gen, hidden=1024, ff=16)
    h = torch.randn(T, 1024, generator=gen).to(DEV, torch.bfloat16)
    assert bool(ops.route_layout_wins(T, 1024, 32, 2)) == bool(two) and (part._one_call(h) is None) == (two is None)
    before = ops.launch_count()
    got = part.forward(h, None)
    counted = ops.launch_count() - before
    args, part._args = part._args, None
    before = ops.launch_count()
    want = part.forward(h, None)
    assert torch.equal(got, want) and counted == ops.launch_count() - before
    ops.raise_on_status(part.ctx.status)
