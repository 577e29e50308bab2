"""Routed experts: every token goes through `top` of `experts` small feed-forwards, chosen by the largest router scores.

A step's (token, rank) assignments are laid out expert by expert on the device, the experts' products run as ONE grouped
product each (up with the activation in its epilogue, then down), and the results are added per token in rank order.
Nothing is read back to the host and every grid depends on the step's shapes alone, so the step can be captured.  The
router's logits are float whatever the compute type; its matrix is kept in float32.  A row's result is a function of that
row alone (each output summed over the inner size in index order), so it does not depend on what else the step holds.

Options of the spec: experts with a gate branch and a clamped activation (gate and up as one grouped product, the
activation a kernel between the two products); scores that are a softmax over all router outputs; a learned bias that
takes part in the choice but not in the weights; a constant on the weights; router outputs that stand for experts without
weights, which return their input (their rows of the grouped products stay empty, and the sum per token takes the input
row in their place); a shared expert that every token passes, whose gate/up product also carries, as one more row of its
matrix, the number per token whose sigmoid multiplies its result; experts with a gate branch and silu; logits with a learned
bias, and weights that are a softmax over the chosen logits only.
"""
from __future__ import annotations

from dataclasses import dataclass
from typing import Dict, List

import torch

from ..csrc import ops
from .context import BuildContext
from .linear import Linear
from .registry import register_feed_forward
from .spec import RoutedExpertsSpec, TensorRole


GATED_EXPERTS = ("glu_clamped", "swiglu")      # activations of experts that have a gate branch


@dataclass
class RoutedRows:
    """The experts' results before they are added up per token: rows [T * top, hidden] float32 laid out expert by expert,
    `row_of[t * top + j]` the row of token t's rank j, `weights` the chosen scores, `scale` whether they still multiply.
    A norm that stands behind the experts adds the rows up itself (`RMSNorm.norm_add`)."""
    rows: torch.Tensor
    row_of: torch.Tensor
    weights: torch.Tensor
    top: int
    scale: bool


@register_feed_forward("routed_experts")
class RoutedExperts:
    @staticmethod
    def expected_tensors(spec: RoutedExpertsSpec) -> List[TensorRole]:
        outputs = spec.experts + spec.identity
        roles = [TensorRole("router.weight", (outputs, spec.hidden), True, True)]
        if spec.choice_bias:
            roles.append(TensorRole("router.bias", (outputs,), role="bias"))
        if spec.logit_bias:
            roles.append(TensorRole("router.logit_bias", (outputs,), role="bias"))
        for e in range(spec.experts):
            if spec.activation in GATED_EXPERTS:
                roles.append(TensorRole(f"experts.{e}.gate.weight", (spec.intermediate, spec.hidden), True, True))
            roles += [TensorRole(f"experts.{e}.up.weight", (spec.intermediate, spec.hidden), True, True),
                      TensorRole(f"experts.{e}.down.weight", (spec.hidden, spec.intermediate), True, True)]
        if spec.shared is not None:
            im = spec.shared.intermediate
            roles += [TensorRole("shared.gate.weight", (im, spec.hidden), True, True),
                      TensorRole("shared.up.weight", (im, spec.hidden), True, True),
                      TensorRole("shared.down.weight", (spec.hidden, im), True, True)]
            if spec.shared.gated:
                roles.append(TensorRole("shared.scale.weight", (1, spec.hidden), True, True))
        return roles

    gives_rows = True          # forward(..., summed=False) hands out RoutedRows (the plain form; the extended one sums itself)

    def __init__(self, spec: RoutedExpertsSpec, tensors: Dict[str, torch.Tensor], ctx: BuildContext):
        self.glu = spec.activation in GATED_EXPERTS
        self.clamped = spec.activation == "glu_clamped"
        if not self.glu and (spec.activation not in ops.EXPERT_ACTIVATIONS or spec.activation == "none"):
            raise ValueError(f"unknown activation '{spec.activation}' of an expert (relu2, {', '.join(GATED_EXPERTS)})")
        if spec.router_activation not in ops.ROUTER_MODES:
            raise ValueError(f"unknown router activation '{spec.router_activation}' ({', '.join(ops.ROUTER_MODES)})")
        outputs = spec.experts + spec.identity
        if spec.experts < 1 or spec.identity < 0 or not 1 <= spec.top <= min(outputs, 32):
            raise ValueError(f"top={spec.top} must be between 1 and the number of router outputs ({outputs}), at most 32")
        if self.clamped and not spec.limit > 0.0:
            raise ValueError("the clamped activation wants a positive limit")
        if spec.shared is not None and not self.glu:
            raise ValueError("a shared expert has the routed experts' form, with a gate branch")
        self.extended = bool(spec.identity or spec.shared is not None or spec.choice_bias or spec.route_scale != 1.0
                             or spec.router_activation in ("softmax", "softmax_chosen") or spec.logit_bias or self.glu)
        if self.extended and spec.scale_input:
            raise ValueError("identity experts, a shared expert and experts with a gate branch weigh the experts' results, not their inputs")
        self.spec, self.ctx = spec, ctx
        f32 = lambda t: t.to(device=ctx.device, dtype=torch.float32).contiguous()
        self.router = f32(tensors["router.weight"])
        self.choice_bias = f32(tensors["router.bias"]) if spec.choice_bias else None
        self.logit_bias = f32(tensors["router.logit_bias"]) if spec.logit_bias else None
        if self.glu:            # gate above up, per expert: one grouped product for both
            self.up = torch.stack([torch.cat([ctx.matrix(tensors[f"experts.{e}.gate.weight"]),
                                              ctx.matrix(tensors[f"experts.{e}.up.weight"])], dim=0)
                                   for e in range(spec.experts)]).contiguous()
        else:
            self.up = torch.stack([ctx.matrix(tensors[f"experts.{e}.up.weight"]) for e in range(spec.experts)]).contiguous()
        self.down = torch.stack([ctx.matrix(tensors[f"experts.{e}.down.weight"]) for e in range(spec.experts)]).contiguous()
        self.tensor_cores = ctx.gemm != "library"
        self.shared_up = self.shared_down = None
        self.shared_block = 0
        if spec.shared is not None:
            if self.clamped and not spec.shared.limit > 0.0:
                raise ValueError("the shared expert's clamped activation wants a positive limit")
            if spec.shared.gated and not self.clamped:
                raise ValueError("a shared expert behind a sigmoid gate has the clamped activation")
            gate, up, im = tensors["shared.gate.weight"], tensors["shared.up.weight"], spec.shared.intermediate
            rows = [gate, up]
            if not self.clamped and im % 64 == 0:      # gate and up in blocks of 64 rows: products with the activation inside take them
                self.shared_block = 64
                rows = [torch.stack([gate.reshape(im // 64, 64, -1), up.reshape(im // 64, 64, -1)], dim=1).reshape(2 * im, -1)]
            if spec.shared.gated:                  # the number per token rides as one more row; zeros up to a multiple of 8 rows
                w = tensors["shared.scale.weight"].reshape(1, -1)
                rows += [w, torch.zeros((7, w.shape[1]), dtype=w.dtype, device=w.device)]
            self.shared_up = Linear(torch.cat(rows, dim=0), None, ctx, label="proj_gate_up")
            self.shared_down = Linear(tensors["shared.down.weight"], None, ctx, label="proj_down")
        self._args, self._scratch, self._counts = self._step_args(outputs), {}, {}      # (sizes by the number of tokens)

    def _step_args(self, outputs: int):
        """The layer as the one-call step takes it (bfloat16, inner sizes of whole 16-byte pieces), or None."""
        s, sh = self.spec, self.spec.shared
        if self.ctx.compute_dtype != torch.bfloat16 or not self.tensor_cores or s.hidden % 8 or s.intermediate % 8 or self.up.dtype != torch.bfloat16:
            return None
        ptr = lambda t: None if t is None else t.data_ptr()
        return ops.ExpertsArgs(
            router=ptr(self.router), choice_bias=ptr(self.choice_bias), logit_bias=ptr(self.logit_bias), up=ptr(self.up), down=ptr(self.down),
            shared_up=ptr(self.shared_up.weight) if sh else None, shared_down=ptr(self.shared_down.weight) if sh else None, status=ptr(self.ctx.status),
            hidden=s.hidden, intermediate=s.intermediate, experts=s.experts, outputs=outputs, top=s.top,
            mode=ops.ROUTER_MODES[s.router_activation], renorm=int(s.renormalize), scale_input=int(s.scale_input),
            act=0 if self.glu else ops.EXPERT_ACTIVATIONS[s.activation], gated=(1 if self.clamped else 2) if self.glu else 0, extended=int(self.extended),
            shared=sh.intermediate if sh else 0, shared_rows=self.shared_up.out_features if sh else 0, shared_block=self.shared_block,
            shared_gated=int(sh.gated) if sh else 0, few=ops.ROUTE_ROWS_TOKENS, route_scale=s.route_scale, limit=s.limit if self.clamped else 0.0,
            shared_limit=sh.limit if sh and self.clamped else 0.0, alpha=1.702)

    def _one_call(self, h: torch.Tensor):
        """The whole step as one call, or None where it does not take the step (or kernel classes are being timed)."""
        if self._args is None or ops.profiling() or h.dtype != torch.bfloat16 or not h.is_contiguous() or h.data_ptr() % 16:
            return None
        T, s = h.shape[0], self.spec
        inside = s.shared is not None and s.shared.intermediate % 8 == 0 and self.shared_up.fuses(T) and self.shared_down.fuses(T)
        size = self._scratch.get(T)
        if size is None:
            if len(self._scratch) >= 4096:
                self._scratch.clear()
            size = self._scratch[T] = ops.experts_scratch(self._args, T, inside)
        if size < 0:                   # asked before the shared expert runs: whoever takes the step then runs it
            return None
        out = torch.empty((T, s.hidden), dtype=torch.float32, device=h.device)
        scratch = torch.empty((size,), dtype=torch.uint8, device=h.device)
        up, down = (self.shared_up.fused_splits(T), self.shared_down.fused_splits(T)) if inside else (0, 0)
        if not ops.experts_step(self._args, h, scratch, out, up, down):
            return None
        if s.shared is not None and not inside:
            ops.experts_sum(self._args, h, scratch, out, *self._shared(h))
        return out

    def _gate(self, gate_up: torch.Tensor, out: torch.Tensor, limit: float, block: int = 0) -> None:
        """The experts' activation: gate_up [rows, >= 2 n] = [gate | up | ...] (or gate and up in turns of `block` columns)
        -> out [rows, n]."""
        if self.clamped:
            ops.glu_clamped(gate_up, out, limit)
        else:
            ops.swiglu(gate_up, out, block)

    def _shared(self, h: torch.Tensor):
        """The shared expert's rows, float32 [T, hidden], and the numbers of its gate [T] (None without one)."""
        s, T = self.spec, h.shape[0]
        im = s.shared.intermediate
        act = self.shared_up.of(h, swiglu=True) if self.shared_block else None
        if act is None:
            # [T, gate | up (| the gate's number, zeros)]: float from the fused product of few rows, else in the compute type
            gu = self.shared_up.full_f32(h) if self.shared_up.fuses(T) else self.shared_up(h)
            act = torch.empty((T, im), dtype=self.ctx.compute_dtype, device=h.device)
            self._gate(gu, act, s.shared.limit, self.shared_block)
        return self.shared_down.full_f32(act), gu[:, 2 * im] if s.shared.gated else None

    def forward(self, h: torch.Tensor, batch, summed: bool = True):
        """h [T, hidden] in the compute type -> the sum of the chosen experts' results, float32 [T, hidden]; or, with
        `summed` False, the results as `RoutedRows`, for a consumer that adds them up itself."""
        if not isinstance(h, torch.Tensor):
            h = h.tensor()
        out = self._one_call(h) if summed or self.extended else None
        if out is not None:
            return out
        s, dev, ct = self.spec, h.device, self.ctx.compute_dtype
        T, A = h.shape[0], h.shape[0] * s.top
        outputs = s.experts + s.identity
        counts = self._counts.get(T)
        if counts is None:
            if len(self._counts) >= 4096:
                self._counts.clear()
            counts = self._counts[T] = ops.route_layout_wins(T, s.hidden, outputs, s.top)
        ints = torch.empty((3 * A + outputs + 1 + counts,), dtype=torch.int32, device=dev)
        ids, row_of, src_of, offsets = ints[:A].view(T, s.top), ints[A:2 * A], ints[2 * A:3 * A], ints[3 * A:3 * A + outputs + 1]
        weights = torch.empty((T, s.top), dtype=torch.float32, device=dev)
        xp = torch.empty((A, s.hidden), dtype=ct, device=dev)
        how = dict(sigmoid=s.router_activation, renorm=s.renormalize, bias=self.choice_bias, scale=s.route_scale, logit_bias=self.logit_bias)
        place = (h, self.router, s.top, ids, weights, offsets, row_of, src_of, xp, s.scale_input)
        if not (ops.route_rows(*place, **how) if T <= ops.ROUTE_ROWS_TOKENS else ops.route_place(*place, ints[3 * A + outputs + 1:] if counts else None, **how)):
            ops.route(h, self.router, s.top, ids, weights, **how)
            ops.route_sort(ids.view(-1), outputs, offsets, row_of, src_of)
            ops.route_gather(h, weights.view(-1), src_of, xp, s.top, scale=s.scale_input)
        if s.identity:                                 # (rows of experts without weights: assigned, never computed)
            offsets = offsets[:s.experts + 1]
        hp = torch.empty((A, s.intermediate), dtype=ct, device=dev)
        if self.glu:
            gu = torch.empty((A, 2 * s.intermediate), dtype=ct, device=dev)
            ops.gemm_grouped(xp, self.up, offsets, gu, "none", self.ctx.status, self.tensor_cores)
            self._gate(gu, hp, s.limit)
        else:
            ops.gemm_grouped(xp, self.up, offsets, hp, s.activation, self.ctx.status, self.tensor_cores)
        yp = torch.empty((A, s.hidden), dtype=torch.float32, device=dev)
        ops.gemm_grouped(hp, self.down, offsets, yp, "none", self.ctx.status, self.tensor_cores)
        if not self.extended:
            if not summed:
                return RoutedRows(yp, row_of, weights.view(-1), s.top, not s.scale_input)
            out = torch.empty((T, s.hidden), dtype=torch.float32, device=dev)
            ops.route_combine(yp, weights.view(-1), row_of, out, s.top, scale=not s.scale_input)
            return out
        shared, gate = self._shared(h) if s.shared is not None else (None, None)
        out = torch.empty((T, s.hidden), dtype=torch.float32, device=dev)
        ops.route_combine_ext(yp, weights.view(-1), row_of, ids.view(-1), s.experts, h, out, s.top, shared=shared, sg=gate)
        return out
