"""Mixture of experts: a grouped top-k router, clamped gated experts, identity outputs and a shared expert.

Steps of ``forward`` (no step waits for the host):

1. router logits in fp32 (one product), then ``ops.moe_route``: softmax over all outputs, the correction for the
   choice only, the best groups, the top-k outputs and their scores as weights;
2. ``ops.moe_group``: the (token, choice) pairs that go to real experts, sorted by expert on the device;
3. two grouped products over that order (``csrc/grouped_gemm.cu``): gate and up with the clamped activation,
   then down into fp32 rows; in bfloat16, when the experts get many rows each (prompts), the rows are gathered
   side by side instead and the two products go to tcgen05 (``csrc/grouped_tcgen05.cu``) over the experts' row ranges, or,
   where that kernel refuses the sizes, every expert's products go through ``linear``, for which the
   host reads the experts' offsets once (the only wait of the part, and never inside a graph capture);
4. ``ops.moe_combine``: each token adds its weighted rows, in the order of its choices, and its own input for
   an identity output;
5. the shared expert, if any: gate/up product, the same activation with its own limit, down with the residual add.

Options of the spec: experts (and the shared one) that are SiLU gates without limits, the same kernels with other
constants; weights divided by their sum and multiplied by a constant (in the routing kernel); sigmoid scores instead of the softmax (a flag of the routing kernel); ungated experts with the
squared ReLU (one up matrix per expert); the activation in the grouped product's epilogue, of many rows on the sums as bfloat16 holds them; weights that multiply the experts' inputs (the rows are gathered in the
sorted order and multiplied by their pair's weight in fp32 on the way, ``ops.moe_gather``; the combine then adds
the chosen rows unweighted).
"""

from __future__ import annotations

import math

import torch

from ..config.specs import RoutedExpertsSpec
from ..kernels import ops
from ..weights.tensors import TensorDecl
from .base import Part, register_part
from .linear import clamped_gated_linear, gated_linear, linear


# From this many rows per expert on (on average) the experts' outputs are rounded to the compute dtype (half the bytes of many rows), and the
# products go to tcgen05 over gathered rows (experts that it refuses one by one through linear(), which waits for the host): neither in a
# step of a graph, whose outputs stay fp32 at any number of rows.  fp32 outputs come from the form that gathers in its loads
# (mma.sync), which sums 16 k inside the tensor core and joins those sums in fp32, where tcgen05 keeps all of K in one sum that cuts off: down
# products of 512 / 1,024 / 2,048 k are 7.1e-8 / 7.6e-8 / 8.2e-8 of their norm from 64 bits, on tcgen05 6.0e-7 / 1.2e-6 / 2.4e-6 (rounded to
# bfloat16 both are 1.7e-3).  What that costs, gather and both products with the weights from memory, us, mma.sync / tcgen05, experts of 2,048 and 1,024:
# 30 of 8 rows 80 / 95, of 16 108 / 95, of 31 170 / 97, four of 30 with all rows 62 / 33, 92 / 37, 157 / 43; 8 experts of 1,024 and 512, 8 rows 18 / 23,
# 31 rows 29 / 24.  tcgen05 for gate and up alone gains nothing (30 x 16 rows 128, 31 rows 168).
# On tcgen05 the first product's sums, like the shared expert's, are rounded before the activation (the bits of a bfloat16 product and an activation
# behind it): layers route by what such rows leave, and sums rounded once, after the activation, moved logits by 0.027 of their norm where two
# scores nearly tied.
ROWS_PER_EXPERT_ROUNDED = 32


def rounds_outputs(dtype: torch.dtype, table: "ops.RoutingTable", ctx) -> bool:
    """Whether the experts' outputs of a step are rounded to the compute dtype before they are combined."""
    return (dtype == torch.bfloat16 and table.n_pairs >= ROWS_PER_EXPERT_ROUNDED * table.n_experts
            and not getattr(ctx, "captured", False) and not torch.cuda.is_current_stream_capturing())


class RoutedExperts(Part):
    graph_safe = True   # the grouped products wait for no one; the per-expert form is not chosen while capturing
    returns_output = True   # forward(..., residual=None) returns the fp32 output instead of adding it

    def __init__(self, spec: RoutedExpertsSpec) -> None:
        super().__init__(spec)
        n_all = spec.num_experts + spec.num_identity
        if spec.num_experts < 0 or spec.num_identity < 0 or n_all <= 0:
            raise ValueError("a router needs at least one output")
        if spec.num_groups <= 0 or n_all % spec.num_groups != 0:
            raise ValueError(f"{n_all} router outputs do not form {spec.num_groups} equal groups")
        if not 0 < spec.keep_groups <= spec.num_groups:
            raise ValueError("keep_groups must be between 1 and the number of groups")
        if not 0 < spec.top_k <= spec.keep_groups * (n_all // spec.num_groups):
            raise ValueError("top_k exceeds the outputs that the kept groups hold")
        if spec.scoring not in ("softmax", "sigmoid"):
            raise ValueError(f"scoring {spec.scoring!r} is not implemented (softmax and sigmoid are)")
        if spec.expert_form not in ("gated_clamp", "gated_silu", "relu2"):
            raise ValueError(f"expert form {spec.expert_form!r} is not implemented (gated_clamp, gated_silu and relu2 are)")
        if spec.weight_on_input and spec.num_identity > 0:
            raise ValueError("identity outputs take their weight on the output")
        self.gated = spec.expert_form != "relu2"
        # the gated activation g sigmoid(alpha g) (u + shift) of clamped g and u; SiLU times up is its form without limits
        silu = spec.expert_form == "gated_silu"
        self.limit, self.shared_limit = (math.inf, math.inf) if silu else (spec.limit, spec.shared_limit)
        self.gate_alpha, self.up_shift = (1.0, 0.0) if silu else (spec.gate_alpha, 1.0)
        self.n_all = n_all

    def tensor_decls(self):
        s = self.spec
        decls = [TensorDecl(s.prefix + "router", (self.n_all, s.hidden_size))]
        if s.has_correction:
            decls.append(TensorDecl(s.prefix + "correction", (self.n_all,), "zeros"))
        halves = ("gate", "up") if self.gated else ("up",)
        for e in range(s.num_experts):
            decls += [TensorDecl(f"{s.prefix}e{e}.{half}", (s.expert_size, s.hidden_size)) for half in halves]
            decls.append(TensorDecl(f"{s.prefix}e{e}.down", (s.hidden_size, s.expert_size)))
        if s.shared_size > 0:
            decls += [TensorDecl(f"{s.prefix}shared.{half}", (s.shared_size, s.hidden_size)) for half in halves]
            decls.append(TensorDecl(s.prefix + "shared.down", (s.hidden_size, s.shared_size)))
        return decls

    def load(self, fetch, runtime) -> None:
        s = self.spec
        self.runtime = runtime
        self.w_router = fetch.matrix(s.prefix + "router")
        self.correction = fetch.vector(s.prefix + "correction") if s.has_correction else None
        halves = ("gate", "up") if self.gated else ("up",)
        if s.num_experts > 0:
            # per expert: gate rows then up rows, so that one grouped product yields both (ungated: the up rows)
            self.w_gate_up = torch.stack([torch.cat([fetch.matrix(f"{s.prefix}e{e}.{half}") for half in halves], 0)
                                          for e in range(s.num_experts)])
            self.w_down = torch.stack([fetch.matrix(f"{s.prefix}e{e}.down") for e in range(s.num_experts)])
            self.counts = torch.zeros(s.num_experts, dtype=torch.int32, device=runtime.device)
        if s.shared_size > 0:
            self.w_shared_gate_up = torch.cat([fetch.matrix(f"{s.prefix}shared.{half}") for half in halves], 0)
            self.w_shared_down = fetch.matrix(s.prefix + "shared.down")

    def forward(self, x, ctx, residual):
        """Adds to ``residual`` (fp32); with ``residual`` None returns the output as a new fp32 tensor."""
        s = self.spec
        n, dev = x.shape[0], x.device
        logits = linear(x, self.w_router, out_dtype=torch.float32)
        ids = torch.empty((n, s.top_k), dtype=torch.int32, device=dev)
        weights = torch.empty((n, s.top_k), dtype=torch.float32, device=dev)
        ops.moe_route(logits, self.correction, ids, weights, n_groups=s.num_groups, keep=s.keep_groups,
                      sigmoid=s.scoring == "sigmoid", renormalise=s.renormalise, scale=s.weight_scale)
        # float32 steps of a few rows per expert: the grouped product that streams weights through registers
        experts = (self.w_gate_up, self.w_down) if s.num_experts > 0 else ()
        few_ok = ops.grouped_few_rows_ok((s.hidden_size, s.expert_size), x.dtype)
        table = ops.RoutingTable(n, s.top_k, max(s.num_experts, 1), dev, few_rows_ok=few_ok,
                                 tensor=ops.grouped_tensor_ok((s.hidden_size, s.expert_size), x.dtype, x, *experts))
        wide_out = lambda: torch.empty((table.n_pairs, s.hidden_size), dtype=torch.float32, device=dev)
        if s.num_experts == 0:
            expert_out = wide_out()                # nobody writes or reads a row of it
        else:
            ops.moe_group(ids, self.counts, table)
            act = torch.empty((table.n_pairs, s.expert_size), dtype=x.dtype, device=dev)
            first_epi = ops.GROUPED_GATED_CLAMP if self.gated else ops.GROUPED_RELU2
            many = rounds_outputs(x.dtype, table, ctx)
            if many and ops.grouped_tcgen05_ok(x.dtype, self.w_gate_up, self.w_down):
                rows = torch.empty((table.n_pairs, s.hidden_size), dtype=x.dtype, device=dev)
                ops.moe_gather(x, table, rows, weights if s.weight_on_input else None)
                ops.grouped_gemm_sorted(rows, self.w_gate_up, act, table.offsets, epi=first_epi, limit=self.limit, alpha=self.gate_alpha,
                                        up_shift=self.up_shift, round_sums=True)
                expert_out = rows           # read by the first product: the outputs, of the same size, take their place
                ops.grouped_gemm_sorted(act, self.w_down, expert_out, table.offsets, epi=ops.GROUPED_STORE)
            elif many:
                expert_out = wide_out()
                self._experts_one_by_one(x, table, act, expert_out, weights)
            elif s.weight_on_input:
                rows, expert_out = torch.empty((table.n_pairs, s.hidden_size), dtype=x.dtype, device=dev), wide_out()
                ops.moe_gather(x, table, rows, weights)
                ops.grouped_gemm_routed(rows, self.w_gate_up, act, table, gather=False, epi=first_epi, limit=self.limit,
                                        alpha=self.gate_alpha, up_shift=self.up_shift)
                ops.grouped_gemm_routed(act, self.w_down, expert_out, table, gather=False, epi=ops.GROUPED_STORE_F32)
            else:
                expert_out = wide_out()
                ops.grouped_gemm_routed(x, self.w_gate_up, act, table, gather=True, epi=first_epi, limit=self.limit,
                                        alpha=self.gate_alpha, up_shift=self.up_shift)
                ops.grouped_gemm_routed(act, self.w_down, expert_out, table, gather=False, epi=ops.GROUPED_STORE_F32)
        out = residual
        if residual is None:       # the caller wants the output itself: the combine assigns, the shared expert adds
            out = torch.empty((n, s.hidden_size), dtype=torch.float32, device=dev)
        ops.moe_combine(out, expert_out, x, ids, None if s.weight_on_input else weights, table, assign=residual is None)
        if s.shared_size > 0:
            if s.expert_form == "gated_silu":
                act = gated_linear(x, self.w_shared_gate_up)
            else:
                act = self._activated(x, self.w_shared_gate_up, self.shared_limit)
            linear(act, self.w_shared_down, residual=out, track=ctx if residual is not None else None)
        return None if residual is not None else out

    def _activated(self, x, weight, limit):
        if self.gated:
            return clamped_gated_linear(x, weight, limit, self.gate_alpha, self.up_shift)
        out = linear(x, weight)
        ops.activation(out, out, "relu2")
        return out

    def _experts_one_by_one(self, x, table, act, expert_out, weights) -> None:
        """The experts' outputs in the sorted order of pairs, into ``expert_out``."""
        s = self.spec
        rows = torch.empty((table.n_pairs, s.hidden_size), dtype=x.dtype, device=x.device)
        ops.moe_gather(x, table, rows, weights if s.weight_on_input else None)
        bounds = table.offsets.tolist()                     # waits for the device
        for e in range(s.num_experts):
            lo, hi = bounds[e], bounds[e + 1]
            if hi > lo:
                act[lo:hi] = self._activated(rows[lo:hi], self.w_gate_up[e], self.limit)
                expert_out[lo:hi].copy_(linear(act[lo:hi], self.w_down[e], out_dtype=torch.float32))


register_part(RoutedExpertsSpec, RoutedExperts)
