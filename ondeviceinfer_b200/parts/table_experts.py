"""Mixture of experts whose choice is a table row per token id, with plain (ungated) experts and a shared expert
that a number per token scales.

Steps of ``forward`` (no step waits for the host):

1. the token's experts are row ``token id`` of the table, each weighted 1 / top;
2. the (token, choice) pairs sorted by expert on the device, with 1 in ``ops.moe_table_group``, once a step;
3. two grouped products over that order (``csrc/grouped_gemm.cu``): up with the activation in its epilogue, then
   down into fp32 rows; in bfloat16, when the experts get many rows each (prompts), the rows are gathered side by
   side and the products go to tcgen05 (``csrc/grouped_tcgen05.cu``) over the experts' row ranges;
4. ``ops.moe_combine``: each token adds its weighted rows in the order of its choices;
5. the shared expert, if any: up, activation, down, added times sigmoid(sg . x): by the kernel of 4, which it then comes before, or by
   ``ops.gated_row_add``.
"""

from __future__ import annotations

import torch

from ..config.specs import TableExpertsSpec
from ..kernels import ops
from ..weights.tensors import TensorDecl
from .base import Part, register_part
from .linear import activated_linear, linear
from .routed_experts import rounds_outputs

GROUPED_EPILOGUE = {"gelu_erf": ops.GROUPED_GELU_ERF, "gelu_tanh": ops.GROUPED_GELU_TANH}


class TableExperts(Part):
    graph_safe = True
    returns_output = True   # forward(..., residual=None) returns the fp32 output instead of adding it

    def __init__(self, spec: TableExpertsSpec) -> None:
        super().__init__(spec)
        if spec.num_experts <= 0 or not 0 < spec.top_k <= spec.num_experts:
            raise ValueError("top_k must be between 1 and the number of experts")
        if spec.activation not in GROUPED_EPILOGUE:
            raise ValueError(f"activation {spec.activation!r} is not implemented ({sorted(GROUPED_EPILOGUE)} are)")

    def tensor_decls(self):
        s = self.spec
        decls = [TensorDecl(s.prefix + "table", (s.vocab_size, s.top_k), f"distinct_below:{s.num_experts}")]
        for e in range(s.num_experts):
            decls += [TensorDecl(f"{s.prefix}e{e}.up", (s.expert_size, s.hidden_size)),
                      TensorDecl(f"{s.prefix}e{e}.down", (s.hidden_size, s.expert_size))]
        if s.shared_size > 0:
            decls += [TensorDecl(s.prefix + "shared.up", (s.shared_size, s.hidden_size)),
                      TensorDecl(s.prefix + "shared.down", (s.hidden_size, s.shared_size))]
            if s.shared_gated:
                decls.append(TensorDecl(s.prefix + "shared.sg", (1, s.hidden_size)))
        return decls

    def load(self, fetch, runtime) -> None:
        s = self.spec
        self.runtime = runtime
        self.table = fetch.integer(s.prefix + "table")
        self.w_up = torch.stack([fetch.matrix(f"{s.prefix}e{e}.up") for e in range(s.num_experts)])
        self.w_down = torch.stack([fetch.matrix(f"{s.prefix}e{e}.down") for e in range(s.num_experts)])
        self.counts = torch.zeros(s.num_experts, dtype=torch.int32, device=runtime.device)
        if s.shared_size > 0:
            self.w_shared_up = fetch.matrix(s.prefix + "shared.up")
            self.w_shared_down = fetch.matrix(s.prefix + "shared.down")
            self.w_shared_gate = fetch.matrix(s.prefix + "shared.sg").reshape(-1).contiguous() if s.shared_gated else None

    def forward(self, x, ctx, residual):
        """Adds to ``residual`` (fp32); with ``residual`` None returns the output as a new fp32 tensor."""
        s = self.spec
        n, dev = x.shape[0], x.device
        few_ok = ops.grouped_few_rows_ok((s.hidden_size, s.expert_size), x.dtype)
        tensor = ops.grouped_tensor_ok((s.hidden_size, s.expert_size), x.dtype, x, self.w_up, self.w_down)

        def route():
            ids = torch.empty((n, s.top_k), dtype=torch.int32, device=dev)
            weights = torch.empty((n, s.top_k), dtype=torch.float32, device=dev)
            table = ops.RoutingTable(n, s.top_k, s.num_experts, dev, few_rows_ok=few_ok, tensor=tensor)
            ops.moe_table_group(self.table, ctx.token_ids, ids, weights, self.counts, table, weight=1.0 / s.top_k)
            return ids, weights, table

        # the tokens alone decide: a layer that a step runs twice is routed once
        ids, weights, table = ctx.memo(("table_routing", self, tensor), route)
        act = torch.empty((table.n_pairs, s.expert_size), dtype=x.dtype, device=dev)
        if rounds_outputs(x.dtype, table, ctx) and ops.grouped_tcgen05_ok(x.dtype, self.w_up, self.w_down):
            rows = torch.empty((table.n_pairs, s.hidden_size), dtype=x.dtype, device=dev)
            ops.moe_gather(x, table, rows)
            ops.grouped_gemm_sorted(rows, self.w_up, act, table.offsets, epi=GROUPED_EPILOGUE[s.activation], round_sums=True)
            expert_out = rows               # read by the first product: the outputs, of the same size, take their place
            ops.grouped_gemm_sorted(act, self.w_down, expert_out, table.offsets, epi=ops.GROUPED_STORE)
        else:
            expert_out = torch.empty((table.n_pairs, s.hidden_size), dtype=torch.float32, device=dev)
            ops.grouped_gemm_routed(x, self.w_up, act, table, gather=True, epi=GROUPED_EPILOGUE[s.activation])
            ops.grouped_gemm_routed(act, self.w_down, expert_out, table, gather=False, epi=ops.GROUPED_STORE_F32)
        assign = residual is None
        if assign:
            residual = torch.empty((n, s.hidden_size), dtype=torch.float32, device=dev)
        gated = s.shared_size > 0 and self.w_shared_gate is not None
        if s.shared_size > 0:
            shared = activated_linear(x, self.w_shared_up, s.activation)
        y = linear(shared, self.w_shared_down, out_dtype=torch.float32) if gated else None
        if gated and ops.moe_combine_gates(x, self.w_shared_gate, residual, expert_out, y):
            ops.moe_combine(residual, expert_out, x, ids, weights, table, assign=assign, shared=(y, self.w_shared_gate))
        else:
            ops.moe_combine(residual, expert_out, x, ids, weights, table, assign=assign)
            if gated:
                ops.gated_row_add(residual, y, x, self.w_shared_gate)
            elif s.shared_size > 0:
                linear(shared, self.w_shared_down, residual=residual)
        if ctx is not None:
            ctx.residual_sumsq = None
        return residual if assign else None


register_part(TableExpertsSpec, TableExperts)
