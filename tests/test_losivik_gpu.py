"""The Losivik design in the engine against its plain restatement (``plain_losivik``): each mechanism alone, whole
prompts, token-by-token decoding, portions, batches of unequal requests, slots and pages used again, far keys, page
borders, the edges of windows and of the kept first positions, the first tokens, long decoding round the ring of a
windowed cache with pinned first pages, sizes off every multiple, and greedy generation through ``generate`` and
the command line.

float32 is compared strictly.  bfloat16 is compared by the error of a row relative to the row's size; where a model
has routed experts a close call of the router may send a row another way than the plain implementation, so the
largest row error is bounded only for models without them."""

import copy
import json
import math
import subprocess
import sys
from pathlib import Path

import pytest
import torch

import ondeviceinfer_b200 as odi
import plain_losivik as plain
from helpers import F32_ATOL, F32_RTOL, write_model_folder
from ondeviceinfer_b200.kernels import ops

pytestmark = pytest.mark.gpu
DTYPES = ["float32", "bfloat16"]
CONFIGS = {"A": (plain.TINY_A, 51), "B": (plain.TINY_B, 52), "C": (plain.TINY_C, 53), "sharp": (plain.SHARP, 54),
           "D": (plain.TINY_D, 55), "E": (plain.TINY_E, 56)}
SHARPEN = {"sharp": 3.0}
_MODELS, _PLAIN = {}, {}


def weights_of(case):
    return plain.random_weights(*CONFIGS[case], sharpen=SHARPEN.get(case, 1.0))


def engine(case, dtype, tmp_path_factory):
    if (case, dtype) not in _MODELS:
        folder = write_model_folder(tmp_path_factory.mktemp(f"losivik_{case}"), CONFIGS[case][0], weights_of(case))
        _MODELS[(case, dtype)] = odi.load_resident_model(folder, dtype=dtype)
    return _MODELS[(case, dtype)]


def expected(case, tokens):
    key = (case, tuple(tokens))
    if key not in _PLAIN:
        _PLAIN[key] = plain.forward(CONFIGS[case][0], weights_of(case), list(tokens)).float()
    return _PLAIN[key]


def routed(cfg):
    return any((layer.get("mlp") or {}).get("kind") == "moe" for layer in cfg["layers"])


def close(actual, reference, dtype, what, atol=None, flips=False):
    """float32: the helpers' strict comparison, or with ``atol`` |d| <= atol.  bfloat16: row error relative to the
    row's size: median at most 2e-2, nine rows in ten within 6e-2, and, unless the router may flip (``flips``), every
    row within 2e-1."""
    if dtype == "float32" and atol is not None:
        gap = float((actual.float().cpu() - reference.float().cpu()).abs().max())
        assert actual.shape == reference.shape and gap <= atol, f"{what}: fp32 max |d| = {gap:.3e}"
        return
    if dtype == "float32":
        # the helpers' bound, which is stated for logits of size one, plus a term for the size of these: the rounding
        # of an fp32 sum grows with its terms, and the tied head of these models gives logits of several tens (observed:
        # up to 5e-6 of the largest logit after three layers with squared activations; one bfloat16 rounding anywhere
        # would show as 1e-3 of it, a key too many or too few as more)
        actual, reference = actual.float().cpu(), reference.float().cpu()
        assert actual.shape == reference.shape and torch.isfinite(actual).all(), what
        gap = (actual - reference).abs()
        bound = F32_ATOL + F32_RTOL * reference.abs() + 1e-5 * float(reference.abs().max())
        assert not (gap > bound).any(), f"{what}: fp32 max |d| = {float(gap.max()):.3e} at logits up to {float(reference.abs().max()):.1f}"
        return
    actual, reference = actual.float().cpu(), reference.float().cpu()
    assert actual.shape == reference.shape and torch.isfinite(actual).all(), what
    error = (actual - reference).norm(dim=-1) / reference.norm(dim=-1).clamp_min(1e-6)
    ranked = error.sort().values
    high = ranked[int(0.9 * len(ranked))] if len(ranked) >= 10 else ranked[-1]
    assert float(error.median()) <= 2e-2 and (float(high) <= 6e-2 or len(ranked) < 10) and (flips or float(ranked[-1]) <= 2e-1), \
        f"{what}: bfloat16 row errors median {float(error.median()):.3e}, high {float(high):.3e}, max {float(ranked[-1]):.3e}"


def ints(*values):
    return torch.tensor(values, dtype=torch.int32, device="cuda")


def tol(dtype):
    return dict(atol=1e-5, rtol=1e-5) if dtype == torch.float32 else dict(atol=2e-2, rtol=2e-2)


# ----------------------------------------------------------------------------- kernels against plain functions


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("width", [6, 7, 64, 200])
def test_scaled_embedding_with_sinusoidal_positions(dtype, width):
    gen = torch.Generator().manual_seed(width)
    table = torch.randn(11, width, generator=gen).to(dtype)
    ids, pos = [3, 0, 10, 3, 7], [0, 1, 2, 700, 4095]
    inv = torch.tensor([10000.0 ** (-2.0 * i / width) for i in range((width + 1) // 2)], dtype=torch.float64).float().cuda()
    out = torch.empty(len(ids), width, device="cuda")
    ops.embed_sinusoid(table.cuda(), ints(*ids), ints(*pos), inv, out, 0.37)
    want = table.double()[ids] * 0.37 + plain.sinusoid(pos, width)
    assert float((out.cpu().double() - want).abs().max()) < 2e-6


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,width", [(1, 4), (5, 37), (9, 192), (3, 2052), (2, 9000)])
def test_two_norms_in_one_pass_and_the_scaled_add(dtype, rows, width):
    gen = torch.Generator().manual_seed(rows * width)
    x = torch.randn(rows, width, generator=gen) * 3
    w1, w2 = torch.randn(width, generator=gen) * 0.2, torch.randn(width, generator=gen) * 0.2
    o1, o2 = torch.empty(rows, width, dtype=dtype, device="cuda"), torch.empty(rows, width, dtype=dtype, device="cuda")
    ops.dual_norm(x.cuda(), (1 + w1).cuda(), (1 + w2).cuda(), 1e-5, o1, o2)
    torch.testing.assert_close(o1.cpu().double(), plain.norm_one_plus(x.double(), w1.double(), 1e-5), **tol(dtype))
    torch.testing.assert_close(o2.cpu().double(), plain.norm_one_plus(x.double(), w2.double(), 1e-5), **tol(dtype))
    a, b = torch.randn(rows, width, generator=gen), torch.randn(rows, width, generator=gen)
    for second in (True, False):
        stream, copy_ = x.clone().cuda(), torch.empty(rows, width, dtype=dtype, device="cuda")
        ops.scaled_add2(stream, a.cuda(), w1.cuda(), b.cuda() if second else None, w2.cuda() if second else None, copy_)
        want = x.double() + a.double() * w1.double() + (b.double() * w2.double() if second else 0)
        torch.testing.assert_close(stream.cpu().double(), want, atol=1e-5, rtol=1e-5)
        torch.testing.assert_close(copy_.cpu().double(), want, **tol(dtype))
    out = torch.empty(rows, width, device="cuda")
    ops.weighted_sum(out, a.cuda(), b.cuda(), 0.6, -1.3)
    torch.testing.assert_close(out.cpu().double(), 0.6 * a.double() - 1.3 * b.double(), atol=1e-5, rtol=1e-5)
    cast = torch.empty(rows, width, dtype=dtype, device="cuda")
    ops.cast_rows(x.cuda(), cast)
    assert torch.equal(cast.cpu(), x.to(dtype))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("dim,layers", [(1, 3), (5, 2), (16, 4)])
def test_gate_times_a_row_picked_by_token_id(dtype, dim, layers):
    gen = torch.Generator().manual_seed(dim)
    z = (torch.randn(7, dim, generator=gen) * 2).to(dtype)
    table = torch.randn(13, dim * layers, generator=gen).to(dtype)
    ids = [12, 0, 5, 5, 1, 9, 12]
    for layer in range(layers):
        out = torch.empty(7, dim, dtype=dtype, device="cuda")
        ops.gated_lookup(z.cuda(), table.cuda(), ints(*ids), out, layer * dim)
        want = plain.gelu_tanh(z.double()) * table.double()[ids][:, layer * dim:(layer + 1) * dim]
        torch.testing.assert_close(out.cpu().double(), want, **tol(dtype))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("d,dv,nq,nkv", [(16, 8, 4, 2), (6, 5, 3, 1), (48, 64, 2, 2), (20, 12, 1, 1), (160, 32, 4, 2)])
def test_head_preparation_with_a_weight_per_lane(dtype, d, dv, nq, nkv):
    gen = torch.Generator().manual_seed(d)
    n, eps = 5, 1e-5
    qkv = torch.randn(n, (nq + nkv) * d + nkv * dv, generator=gen).to(dtype)
    qw, kw = 1 + 0.3 * torch.randn(d, generator=gen), 1 + 0.3 * torch.randn(d, generator=gen)
    lanes = -(-d // 4) * 4
    q_out = torch.empty(n, nq * lanes, dtype=dtype, device="cuda")
    k_pool = torch.zeros(2, nkv, 64, lanes, dtype=dtype, device="cuda")
    v_pool = torch.zeros(2, nkv, 64, dv, dtype=dtype, device="cuda")
    pos = [62, 63, 64, 65, 66]       # over a page border
    ops.rot_unit_prep(qkv.cuda(), q_out, k_pool, v_pool, None, None, ints(0, 0, 0, 0, 0), ints(*pos), ints(0, 2), ints(1, 0),
                      nq=nq, nkv=nkv, d=d, dv=dv, rot_dim=0, page_size=64, ring_pages=0, write_kv=True, unit_eps=eps,
                      d_store=lanes, q_weight=qw.cuda(), k_weight=kw.cuda())
    x = qkv.double()
    want_q = plain.norm_plain(x[:, :nq * d].view(n, nq, d), qw.double(), eps)
    want_k = plain.norm_plain(x[:, nq * d:(nq + nkv) * d].view(n, nkv, d), kw.double(), eps)
    want_v = x[:, (nq + nkv) * d:].view(n, nkv, dv)
    torch.testing.assert_close(q_out.cpu().double().view(n, nq, lanes)[:, :, :d], want_q, **tol(dtype))
    assert float(q_out.cpu().double().view(n, nq, lanes)[:, :, d:].abs().sum()) == 0
    for i, p in enumerate(pos):
        page = [1, 0][p // 64]
        torch.testing.assert_close(k_pool[page, :, p % 64, :d].cpu().double(), want_k[i], **tol(dtype))
        torch.testing.assert_close(v_pool[page, :, p % 64].cpu().double(), want_v[i], **tol(dtype))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_head_gate_with_one_number_per_head(dtype):
    gen = torch.Generator().manual_seed(3)
    for heads, dv, lanes in ((3, 5, 5), (4, 16, 32), (1, 8, 8)):
        x = torch.randn(6, heads * lanes, generator=gen).to(dtype)
        gate = torch.randn(6, 10 + heads, generator=gen).to(dtype)
        got = x.clone().cuda()
        ops.gate_heads(got, gate.cuda(), heads=heads, dv=dv, lanes=lanes, col=10, per_head=True)
        want = x.double().view(6, heads, lanes).clone()
        want[:, :, :dv] *= torch.sigmoid(gate.double()[:, 10:])[:, :, None]
        torch.testing.assert_close(got.cpu().double().view(6, heads, lanes), want, **tol(dtype))


def test_router_with_sigmoid_scores_against_the_plain_choice():
    gen = torch.Generator().manual_seed(5)
    for n_experts, top in ((8, 1), (5, 3), (3, 3), (40, 4)):
        logits = torch.randn(33, n_experts, generator=gen) * 2
        logits[4] = 0.25                      # all equal: the lowest indices win
        logits[5, 1] = logits[5, 2] = 3.0     # a tie at the top
        ids = torch.empty(33, top, dtype=torch.int32, device="cuda")
        weights = torch.empty(33, top, dtype=torch.float32, device="cuda")
        ops.moe_route(logits.cuda(), None, ids, weights, n_groups=1, keep=1, sigmoid=True)
        chosen, scores = plain.router_choice({"router": torch.eye(n_experts, dtype=torch.float64)}, "", {"router": {"top": top}},
                                             logits.double())
        assert torch.equal(ids.cpu().long(), chosen)
        torch.testing.assert_close(weights.cpu().double(), scores, atol=1e-6, rtol=1e-6)


# whole tiles of rows (each expert gets every token), fewer rows than tcgen05 takes, more tokens than a fused epilogue takes
@pytest.mark.parametrize("n", [8, 64, 1024])
def test_activations_are_of_the_products_as_bfloat16_holds_them(n):
    """Ungated experts of many rows, their shared expert and the clamped gated feed-forward: the activation of the rounded product, bit for
    bit; with few rows an expert the sums of the grouped product that gathers in its loads, as they are."""
    from ondeviceinfer_b200.config.specs import ClampedGatedMLPSpec, RoutedExpertsSpec
    from ondeviceinfer_b200.parts import Runtime, build_part
    from ondeviceinfer_b200.parts.linear import linear
    gen = torch.Generator().manual_seed(n)
    H, F, E = 128, 64, 2
    matrix = lambda *shape: (torch.randn(*shape, generator=gen) / math.sqrt(shape[-1])).bfloat16().cuda()
    x = torch.randn(n, H, generator=gen).bfloat16().cuda()
    runtime = Runtime(dtype=torch.bfloat16, device=torch.device("cuda"))
    mlp = build_part(ClampedGatedMLPSpec(hidden_size=H, intermediate_size=F, prefix="", limit=1.5, alpha=1.2,
                                         names=(("gate", "gate"), ("up", "up"), ("down", "down"))))
    experts = build_part(RoutedExpertsSpec(hidden_size=H, expert_size=F, num_experts=E, num_identity=0, top_k=E, num_groups=1, keep_groups=1,
                                           limit=0.0, prefix="", has_correction=False, shared_size=F, scoring="sigmoid", expert_form="relu2",
                                           weight_on_input=True))
    for part in (mlp, experts):
        w = {d.name: matrix(*d.shape) for d in part.tensor_decls()}
        part.load(type("Fetch", (), {"matrix": staticmethod(w.__getitem__), "vector": staticmethod(w.__getitem__)}), runtime)
    act = torch.empty(n, F, dtype=torch.bfloat16, device="cuda")
    ops.gated_clamp(linear(x, mlp.w_gate_up), act, 1.5, 1.2)
    assert torch.equal(mlp.forward(x, None, None), linear(act, mlp.w_down, out_dtype=torch.float32))

    ids, weights = torch.empty(n, E, dtype=torch.int32, device="cuda"), torch.empty(n, E, device="cuda")
    ops.moe_route(linear(x, experts.w_router, out_dtype=torch.float32), None, ids, weights, n_groups=1, keep=1, sigmoid=True)
    table = ops.RoutingTable(n, E, E, "cuda", tensor=ops.grouped_tensor_ok((H, F), torch.bfloat16, x, experts.w_gate_up, experts.w_down))
    ops.moe_group(ids, experts.counts, table)
    rows, act = (torch.empty(n * E, width, dtype=torch.bfloat16, device="cuda") for width in (H, F))
    ops.moe_gather(x, table, rows, weights)
    if n >= 32:
        ops.grouped_gemm_sorted(rows, experts.w_gate_up, act, table.offsets, epi=ops.GROUPED_STORE)
        ops.activation(act, act, "relu2")
        out = torch.empty(n * E, H, dtype=torch.bfloat16, device="cuda")
        ops.grouped_gemm_sorted(act, experts.w_down, out, table.offsets, epi=ops.GROUPED_STORE)
    else:
        ops.grouped_gemm_routed(rows, experts.w_gate_up, act, table, gather=False, epi=ops.GROUPED_RELU2)
        out = torch.empty(n * E, H, device="cuda")
        ops.grouped_gemm_routed(act, experts.w_down, out, table, gather=False, epi=ops.GROUPED_STORE_F32)
    want = torch.empty(n, H, device="cuda")
    ops.moe_combine(want, out, x, ids, None, table, assign=True)
    shared = linear(x, experts.w_shared_gate_up)
    ops.activation(shared, shared, "relu2")
    linear(shared, experts.w_shared_down, residual=want)
    assert torch.equal(experts.forward(x, None, None), want)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n,H,F,n_experts,top", [(1, 16, 8, 3, 2), (9, 40, 24, 5, 3), (300, 64, 32, 4, 1)])
def test_ungated_experts_with_weights_on_their_inputs(dtype, n, H, F, n_experts, top):
    gen = torch.Generator().manual_seed(n)
    x = torch.randn(n, H, generator=gen).to(dtype)
    up = (torch.randn(n_experts, F, H, generator=gen) / math.sqrt(H)).to(dtype)
    down = (torch.randn(n_experts, H, F, generator=gen) / math.sqrt(F)).to(dtype)
    logits = torch.randn(n, n_experts, generator=gen)
    ids = torch.empty(n, top, dtype=torch.int32, device="cuda")
    weights = torch.empty(n, top, dtype=torch.float32, device="cuda")
    ops.moe_route(logits.cuda(), None, ids, weights, n_groups=1, keep=1, sigmoid=True)
    table = ops.RoutingTable(n, top, n_experts, "cuda", tensor=ops.grouped_tensor_ok((H, F), dtype))
    counts = torch.zeros(n_experts, dtype=torch.int32, device="cuda")
    ops.moe_group(ids, counts, table)
    rows = torch.empty(n * top, H, dtype=dtype, device="cuda")
    ops.moe_gather(x.cuda(), table, rows, weights)
    act = torch.empty(n * top, F, dtype=dtype, device="cuda")
    ops.grouped_gemm_routed(rows, up.cuda(), act, table, gather=False, epi=ops.GROUPED_RELU2)
    out = torch.empty(n * top, H, dtype=torch.float32, device="cuda")
    ops.grouped_gemm_routed(act, down.cuda(), out, table, gather=False, epi=ops.GROUPED_STORE_F32)
    total = torch.zeros(n, H, device="cuda")
    ops.moe_combine(total, out, x.cuda(), ids, None, table)
    want = torch.zeros(n, H, dtype=torch.float64)
    for t in range(n):
        for k in range(top):
            e = int(ids[t, k])
            w = {"up": up[e].double(), "down": down[e].double()}
            want[t] += plain.squared_relu_expert(w, "", (weights[t, k].double().cpu() * x[t].double())[None])[0]
    torch.testing.assert_close(total.cpu().double(), want, **(dict(atol=2e-5, rtol=2e-5) if dtype == torch.float32 else dict(atol=6e-2, rtol=6e-2)))
    flat = torch.randn(50, generator=gen).to(dtype)
    got = torch.empty(50, dtype=dtype, device="cuda")
    ops.activation(flat.cuda(), got, "relu2")
    torch.testing.assert_close(got.cpu().double(), torch.relu(flat.double()) ** 2, **tol(dtype))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("heads,P,N,G,taps,parts", [(4, 32, 48, 2, 3, 2), (3, 5, 10, 1, 1, 3), (6, 16, 24, 3, 4, 1),
                                                     (2, 40, 130, 2, 2, 5), (1, 70, 7, 1, 6, 1)])
def test_state_space_mixer_over_cut_sequences(dtype, heads, P, N, G, taps, parts):
    """Three sequences cut into unequal runs (one token, fewer tokens than taps, more than a staged chunk), stepped
    together with the state carried in slots of their own, against the recurrence over each whole sequence."""
    gen = torch.Generator().manual_seed(heads * P + N)
    inner, C = heads * P, heads * P + 2 * G * N
    M = inner + C + heads
    lengths = [45, 3, 21]
    projs = [(torch.randn(L, M, generator=gen)).to(dtype) for L in lengths]
    w = {"in": torch.eye(M, dtype=torch.float64), "o": torch.eye(inner, dtype=torch.float64),
         "conv": torch.randn(C, taps, generator=gen) * 0.5, "conv.b": torch.randn(C, generator=gen) * 0.1,
         "dt_bias": torch.randn(heads, generator=gen) * 0.5 - 1, "A_log": torch.log(0.05 + torch.rand(heads, generator=gen)),
         "D": 1 + 0.3 * torch.randn(heads, generator=gen), "norm": 1 + 0.1 * torch.randn(inner, generator=gen)}
    m = {"heads": heads, "vdim": P, "state": N, "groups": G, "conv": taps, "norm_groups": parts}
    want = [plain.state_space({k: v.double() for k, v in w.items()}, "", m, p.double(), 1e-5) for p in projs]
    dev = {k: v.float().cuda() for k, v in w.items()}
    slots = [4, 0, 2]
    state = torch.zeros(6, heads, N, P, device="cuda")
    conv_state = torch.zeros(6, taps - 1, C, device="cuda") if taps > 1 else None
    state[1].fill_(7.0)          # a slot of somebody else: must stay as it is
    cuts = [[1, 1, 20, 2, 21], [1, 1, 1], [17, 1, 3]]
    got = [[] for _ in lengths]
    at = [0, 0, 0]
    for step in range(5):
        live = [s for s in range(3) if step < len(cuts[s])]
        runs = [projs[s][at[s]:at[s] + cuts[s][step]] for s in live]
        proj = torch.cat(runs).cuda()
        cu = [0]
        for r in runs:
            cu.append(cu[-1] + len(r))
        tok_seq = [i for i, r in enumerate(runs) for _ in range(len(r))]
        out = torch.empty(proj.shape[0], inner, dtype=dtype, device="cuda")
        ops.ssd_mix(proj, dev["conv"], dev["conv.b"], dev["dt_bias"], dev["A_log"], dev["D"], dev["norm"], conv_state, state, out,
                    ints(*cu), ints(*tok_seq), ints(*[slots[s] for s in live]), n_seqs=len(live), heads=heads, head_dim=P,
                    state_dim=N, groups=G, norm_groups=parts, eps=1e-5)
        for i, s in enumerate(live):
            got[s].append(out[cu[i]:cu[i + 1]].cpu())
            at[s] += cuts[s][step]
    assert float((state[1] - 7.0).abs().max()) == 0
    for s in range(3):
        torch.testing.assert_close(torch.cat(got[s]).double(), want[s], **(dict(atol=2e-4, rtol=2e-4) if dtype == torch.float32
                                                                           else dict(atol=3e-2, rtol=3e-2)))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("heads,P,N,G,taps,parts", [(4, 64, 128, 2, 4, 1), (3, 20, 64, 1, 1, 3), (2, 100, 192, 2, 2, 1)])
def test_state_space_scan_in_chunks_of_tokens(dtype, heads, P, N, G, taps, parts):
    """Runs around the chunks' edges, one of a single token among them, continued by a second step, with decays down to
    those that wipe the state; against the recurrence over each whole sequence, and no further off than the token by token
    kernel.  A token that is not a number reaches no token before it."""
    gen = torch.Generator().manual_seed(heads * P + N)
    inner, C = heads * P, heads * P + 2 * G * N
    M, slots, cuts = inner + C + heads, [3, 0, 4, 1], [[890, 64, 1, 70], [63, 129, 800, 75]]
    lengths = [a + b for a, b in zip(*cuts)]
    projs = [torch.randn(L, M, generator=gen).to(dtype) for L in lengths]
    projs[0][40:42, -heads:] = 300.0             # the state is wiped inside a chunk
    w = {"in": torch.eye(M, dtype=torch.float64), "o": torch.eye(inner, dtype=torch.float64),
         "conv": torch.randn(C, taps, generator=gen) * 0.5, "conv.b": torch.randn(C, generator=gen) * 0.1,
         "dt_bias": torch.randn(heads, generator=gen) * 0.5 - 2, "A_log": torch.log(0.02 + 4 * torch.rand(heads, generator=gen)),
         "D": 1 + 0.3 * torch.randn(heads, generator=gen), "norm": 1 + 0.1 * torch.randn(inner, generator=gen)}
    m = {"heads": heads, "vdim": P, "state": N, "groups": G, "conv": taps, "norm_groups": parts}
    want = [plain.state_space({k: v.double() for k, v in w.items()}, "", m, p.double(), 1e-5) for p in projs]
    dev = {k: v.float().cuda() for k, v in w.items()}

    def run(projs, in_chunks):
        state = torch.zeros(6, heads, N, P, device="cuda")
        conv_state = torch.zeros(6, taps - 1, C, device="cuda") if taps > 1 else None
        state[2].fill_(7.0)          # a slot of somebody else: must stay as it is
        got, at = [[] for _ in lengths], [0] * len(lengths)
        for lens in cuts:
            cu = [0]
            for n in lens:
                cu.append(cu[-1] + n)
            out = torch.empty(cu[-1], inner, dtype=dtype, device="cuda")
            ops.ssd_mix(torch.cat([x[o:o + n] for x, o, n in zip(projs, at, lens)]).cuda(), dev["conv"], dev["conv.b"], dev["dt_bias"],
                        dev["A_log"], dev["D"], dev["norm"], conv_state, state, out, ints(*cu),
                        ints(*[s for s, n in enumerate(lens) for _ in range(n)]), ints(*slots), n_seqs=len(lens), heads=heads, head_dim=P,
                        state_dim=N, groups=G, norm_groups=parts, eps=1e-5, in_chunks=in_chunks)
            for s, n in enumerate(lens):
                got[s].append(out[cu[s]:cu[s + 1]].cpu().double())
                at[s] += n
        assert at == lengths and bool((state[2] == 7.0).all())
        return [torch.cat(g) for g in got], state

    off = lambda got: [float((a - b).norm() / b.norm()) for a, b in zip(got, want)]
    assert ops.ssd_chunk_floats(sum(cuts[0]), 4, heads, P, N, G) > 0
    (chunked, state), (single, state_single) = run(projs, True), run(projs, False)
    rounding = 0.0 if dtype == torch.float32 else 2.0 ** -9      # of the output; all before it is fp32 in both
    assert max(off(chunked)) < rounding + 5e-6 and max(off(single)) < rounding + 5e-6      # sums of a few hundred products of 2^-24 each
    assert sum(off(chunked)) <= (1.25 if dtype == torch.float32 else 1.01) * sum(off(single))
    torch.testing.assert_close(state, state_single, atol=2e-5, rtol=2e-5)
    broken = [p.clone() for p in projs]
    broken[0][100, inner:] = math.nan      # in the middle of a chunk
    got = run(broken, True)[0][0]
    assert bool(torch.equal(got[:100], chunked[0][:100])) and not bool(torch.isfinite(got[100:]).any())


def test_chunks_leave_states_no_further_off_than_token_by_token():
    """The state behind 1,100 tokens, against the recurrence in 64 bits, three seeds together."""
    heads, P, N, T, off = 8, 32, 64, 1100, {True: 0.0, False: 0.0}
    inner, C = heads * P, heads * P + 2 * N
    for seed in range(3):
        gen = torch.Generator().manual_seed(seed)
        proj, conv, conv_b = torch.randn(T, inner + C + heads, generator=gen), torch.randn(C, 4, generator=gen) * 0.3, torch.zeros(C)
        dt_bias, a_log = torch.randn(heads, generator=gen) * 0.5 - 2, torch.log(0.02 + 4 * torch.rand(heads, generator=gen))
        xbc = plain.silu(plain.causal_convolution(proj[:, inner:inner + C].double(), conv.double(), conv_b.double()))
        dt = torch.nn.functional.softplus(proj[:, inner + C:].double() + dt_bias.double())
        keep, S = torch.exp(-torch.exp(a_log.double()) * dt), torch.zeros(heads, N, P, dtype=torch.float64)
        for t in range(T):
            written = xbc[t, inner:inner + N, None] * xbc[t, :inner].view(heads, 1, P)
            S = keep[t, :, None, None] * S + dt[t, :, None, None] * written
        for in_chunks in off:
            state = torch.zeros(1, heads, N, P, device="cuda")
            ops.ssd_mix(proj.cuda(), conv.cuda(), conv_b.cuda(), dt_bias.cuda(), a_log.cuda(), torch.ones(heads, device="cuda"),
                        torch.ones(inner, device="cuda"), torch.zeros(1, 3, C, device="cuda"), state, torch.empty(T, inner, device="cuda"), ints(0, T),
                        ints(*[0] * T), ints(0), n_seqs=1, heads=heads, head_dim=P, state_dim=N, groups=1, norm_groups=1, eps=1e-5,
                        in_chunks=in_chunks)
            off[in_chunks] += float((state[0].cpu().double() - S).norm() / S.norm())
    assert off[True] <= off[False]      # 0.95 of it; with products of decays rounded at every step 1.06


def test_float32_state_space_mixer_depends_on_neither_the_batch_nor_the_cut():
    """A run of 1,100 tokens alone, beside others, and in passes: the same bits."""
    heads, P, N, lens = 2, 64, 64, [1100, 1, 70, 3]
    gen = torch.Generator().manual_seed(6)
    inner, C = heads * P, heads * P + 2 * N
    proj = torch.randn(sum(lens), inner + C + heads, generator=gen).cuda()
    conv, conv_b = (torch.randn(C, 4, generator=gen) * 0.5).cuda(), (torch.randn(C, generator=gen) * 0.1).cuda()
    dt_bias, a_log, skip = (torch.randn(heads, generator=gen).cuda() for _ in range(3))
    norm = torch.ones(inner, device="cuda")

    def run(passes):      # each a list of (sequence, first token, tokens)
        state, conv_state = torch.zeros(4, heads, N, P, device="cuda"), torch.zeros(4, 3, C, device="cuda")
        got = []
        for runs in passes:
            rows = torch.cat([torch.arange(sum(lens[:s]) + first, sum(lens[:s]) + first + n) for s, first, n in runs]).cuda()
            cu = [sum(n for _, _, n in runs[:i]) for i in range(len(runs) + 1)]
            out = torch.empty(cu[-1], inner, device="cuda")
            ops.ssd_mix(proj[rows], conv, conv_b, dt_bias, a_log, skip, norm, conv_state, state, out, ints(*cu),
                        ints(*[i for i, r in enumerate(runs) for _ in range(r[2])]), ints(*[r[0] for r in runs]), n_seqs=len(runs),
                        heads=heads, head_dim=P, state_dim=N, groups=1, norm_groups=1, eps=1e-5)
            got += [out[cu[i]:cu[i + 1]] for i, r in enumerate(runs) if r[0] == 0]
        return torch.cat(got), state[0]

    alone, state = run([[(0, 0, 1100)]])
    for passes in ([[(0, 0, 1100), (1, 0, 1), (2, 0, 70), (3, 0, 3)]], [[(0, 0, 555)], [(2, 0, 70), (0, 555, 544)], [(0, 1099, 1)]]):
        got, end = run(passes)
        assert torch.equal(got, alone) and torch.equal(end, state)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("heads,P,N,lens", [(4, 20, 32, [16]), (16, 64, 64, [460]), (16, 64, 64, [17, 203, 40, 1, 99, 120]), (32, 64, 128, [8, 226])])
def test_convolution_in_pieces_of_eight_tokens(dtype, heads, P, N, lens):
    """Steps below and above the number of inputs from which the convolution takes eight tokens at a time: runs that begin, end and
    meet anywhere in a piece, behind three earlier tokens of theirs; the same bits as token by token."""
    gen = torch.Generator().manual_seed(sum(lens))
    inner, C, n = heads * P, heads * P + 2 * N, sum(lens)
    proj = torch.randn(n, inner + C + heads, generator=gen).to(dtype).cuda()
    conv, conv_b = (torch.randn(C, 4, generator=gen) * 0.5).cuda(), (torch.randn(C, generator=gen) * 0.1).cuda()
    dt_bias, a_log, skip = (torch.randn(heads, generator=gen).cuda() for _ in range(3))
    norm, before = torch.ones(inner, device="cuda"), torch.randn(len(lens), 3, C, generator=gen).cuda()
    starts = [sum(lens[:s]) for s in range(len(lens))]

    def run(steps):      # each a list of (sequence, first token, tokens)
        state, conv_state = torch.zeros(len(lens), heads, N, P, device="cuda"), before.clone()
        got = torch.empty(n, inner, dtype=dtype, device="cuda")
        for runs in steps:
            rows = torch.cat([torch.arange(starts[s] + first, starts[s] + first + m) for s, first, m in runs]).cuda()
            cu = [sum(m for _, _, m in runs[:i]) for i in range(len(runs) + 1)]
            out = torch.empty(cu[-1], inner, dtype=dtype, device="cuda")
            ops.ssd_mix(proj[rows], conv, conv_b, dt_bias, a_log, skip, norm, conv_state, state, out, ints(*cu),
                        ints(*[i for i, r in enumerate(runs) for _ in range(r[2])]), ints(*[r[0] for r in runs]), n_seqs=len(runs),
                        heads=heads, head_dim=P, state_dim=N, groups=1, norm_groups=1, eps=1e-5, in_chunks=False)
            got[rows] = out
        return got, conv_state

    whole, end = run([[(s, 0, m) for s, m in enumerate(lens)]])
    single, end_single = run([[(s, t, 1) for s, m in enumerate(lens) if t < m] for t in range(max(lens))])
    assert torch.equal(whole, single) and torch.equal(end, end_single)


# ----------------------------------------------------------------------------- attention with kept first positions


def _pools(keys, values, ring, pinned, n_extra_pages=3):
    """Pages as a cache with `pinned` first pages and a ring of `ring` pages behind them would hold them after
    writing positions 0..L-1 in order (ring 0: every page kept).  Returns (k_pool, v_pool, page list)."""
    L, nkv, d = keys.shape
    dv = values.shape[-1]
    n_pages = -(-L // 64) if ring == 0 else min(-(-L // 64), pinned + ring)
    order = torch.randperm(n_pages + n_extra_pages).tolist()[:n_pages]
    k_pool = torch.full((n_pages + n_extra_pages, nkv, 64, d), 9.0, dtype=keys.dtype)      # what nobody wrote is loud
    v_pool = torch.full((n_pages + n_extra_pages, nkv, 64, dv), 9.0, dtype=values.dtype)
    for pos in range(L):
        page = pos // 64
        entry = page if ring == 0 or page < pinned else pinned + (page - pinned) % ring
        k_pool[order[entry], :, pos % 64] = keys[pos]
        v_pool[order[entry], :, pos % 64] = values[pos]
    return k_pool.cuda(), v_pool.cuda(), order


def _attention_with_kept_keys(kind, q, keys, values, scale, window, keep, past, ring=0, pinned=0, splits=1):
    T, nq, d = q.shape
    nkv, dv = keys.shape[1], values.shape[-1]
    k_pool, v_pool, pages = _pools(keys, values, ring, pinned)
    out = torch.empty(T, nq * dv, dtype=q.dtype, device="cuda")
    code = pinned * 65536 + ring
    partial = torch.empty(T * nq * splits * (dv + 2), device="cuda") if splits > 1 else None
    args = (q.reshape(T, nq * d).cuda(), k_pool, v_pool, out, ints(0, T), ints(past), ints(0, len(pages)), ints(*pages))
    if kind == "cores":
        ops.attention_simt(*args, n_seqs=1, max_q_len=T, nq=nq, nkv=nkv, d=d, dv=dv, page_size=64, ring_pages=code,
                           window=window, scale=scale, splits=splits, partial=partial, keep=keep)
    elif kind == "tensor":
        ops.attention_capped(*args, n_seqs=1, max_q_len=T, nq=nq, nkv=nkv, d=d, dv=dv, page_size=64, ring_pages=code,
                             window=window, scale=scale, keep=keep)
    elif kind == "tensor memory":
        ops.attention_tcgen05(*args, n_seqs=1, max_q_len=T, nq=nq, nkv=nkv, d=d, page_size=64, ring_pages=code,
                              window=window, scale=scale, keep=keep)
    else:
        ops.attention_capped_decode(*args, n_seqs=1, nq=nq, nkv=nkv, d=d, dv=dv, page_size=64, ring_pages=code, window=window,
                                    scale=scale, splits=splits, partial=partial, keep=keep)
    return out.cpu().view(T, nq, dv)


KEPT_CASES = [  # window, keep, total length, tokens of the step, ring pages, pinned pages, splits
    (40, 5, 150, 150, 0, 0, 1), (40, 5, 150, 1, 0, 0, 1), (40, 5, 150, 1, 0, 0, 3), (30, 70, 300, 60, 3, 2, 1),
    (30, 70, 300, 1, 3, 2, 2), (64, 64, 200, 7, 0, 0, 1), (64, 65, 400, 1, 3, 2, 4), (129, 1, 500, 100, 5, 1, 1),
    (1, 3, 90, 90, 0, 0, 1), (100, 0, 260, 1, 4, 0, 2), (17, 9, 20, 20, 0, 0, 1), (50, 200, 120, 30, 0, 0, 1)]


@pytest.mark.parametrize("kind,dtype", [("cores", torch.float32), ("cores", torch.bfloat16), ("tensor", torch.bfloat16),
                                        ("decode", torch.bfloat16), ("tensor memory", torch.bfloat16)])
@pytest.mark.parametrize("window,keep,L,T,ring,pinned,splits", KEPT_CASES)
def test_attention_that_keeps_the_first_positions(kind, dtype, window, keep, L, T, ring, pinned, splits):
    """Against the plain masked softmax, on pages laid out as the cache lays them out (positions that left the ring are
    overwritten).  One query head asks sharply for the oldest key of its window, one for the key just outside it, one
    for the last kept position and one for the first position that is not kept: a key dropped or kept by mistake moves
    the output by the size of a value."""
    if kind == "decode" and T != 1 or kind in ("tensor", "tensor memory") and splits > 1:
        pytest.skip("the single-token form takes one token; the forms for prompts do not cut the keys")
    gen = torch.Generator().manual_seed(window * 1000 + keep + L)
    nq, nkv, d, dv = (4, 2, 64, 64) if kind == "tensor memory" else (4, 2, 32, 16)
    keys = torch.randn(L, nkv, d, generator=gen)
    keys = keys / keys.norm(dim=-1, keepdim=True)
    values = torch.randn(L, nkv, dv, generator=gen)
    past = L - T
    q = torch.randn(T, nq, d, generator=gen) * 0.3
    for i in range(T):
        p = past + i
        targets = [p - window + 1, p - window, keep - 1, keep]        # in, out, kept, not kept
        for h, target in enumerate(targets):
            if 0 <= target <= p:
                q[i, h] += 40.0 * keys[target, h // (nq // nkv)]
    q, keys, values = q.to(dtype), keys.to(dtype), values.to(dtype)
    got = _attention_with_kept_keys(kind, q, keys, values, 1.0, window, keep, past, ring, pinned, splits)
    seen = plain.visible(L, window, keep)[past:]
    scores = torch.einsum("phd,jhd->hpj", q.double(), keys.double().repeat_interleave(nq // nkv, 1))
    scores = scores.masked_fill(~seen[None], float("-inf"))
    want = torch.einsum("hpj,jhd->phd", torch.softmax(scores, -1), values.double().repeat_interleave(nq // nkv, 1))
    bound = 1e-4 if dtype == torch.float32 else 4e-2
    assert float((got.double() - want).abs().max()) < bound
    # the setup shows a window that is one off, or a kept position too many or too few
    for other in ((window + 1, keep), (window, keep + 1), (window, max(keep - 1, 0))):
        if other == (window, keep):
            continue
        moved = plain.visible(L, *other)[past:]
        if not torch.equal(moved, seen):
            s2 = torch.einsum("phd,jhd->hpj", q.double(), keys.double().repeat_interleave(nq // nkv, 1)).masked_fill(~moved[None], float("-inf"))
            w2 = torch.einsum("hpj,jhd->phd", torch.softmax(s2, -1), values.double().repeat_interleave(nq // nkv, 1))
            assert float((w2 - want).abs().max()) > 0.1


# ----------------------------------------------------------------------------- whole models


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("case", ["A", "B", "C", "D", "E"])
def test_whole_prompts_and_their_first_tokens(case, dtype, tmp_path_factory):
    model = engine(case, dtype, tmp_path_factory)
    cfg = CONFIGS[case][0]
    cache = model.make_cache(max_tokens=512, max_seqs=2)
    for n in (1, 2, 3, 150):
        tokens = plain.random_prompts(cfg, [n], n)[0]
        slot = cache.alloc()
        got = model.step(cache, [slot], [tokens], "all")
        cache.free(slot)
        if n >= 10 or dtype == "float32":
            close(got, expected(case, tokens), dtype, f"{case} whole prompt of {n}", flips=routed(cfg))
    cache.check()


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("case", ["A", "B"])
def test_residual_stream_after_every_layer(case, dtype, tmp_path_factory):
    model = engine(case, dtype, tmp_path_factory)
    cfg = CONFIGS[case][0]
    tokens = plain.random_prompts(cfg, [40], 2)[0]
    want = plain.forward(cfg, weights_of(case), tokens, keep_layers=True)[1].float()
    seen, blocks = [], list(model.decoder.layers)
    originals = [block.forward for block in blocks]
    try:
        for block, original in zip(blocks, originals):
            def record(hidden, ctx, view, original=original):
                result = original(hidden, ctx, view)
                seen.append(hidden.clone())
                return result
            block.forward = record
        cache = model.make_cache(max_tokens=64, max_seqs=1)
        model.step(cache, [cache.alloc()], [tokens], "last")
    finally:
        for block, original in zip(blocks, originals):
            block.forward = original
    assert len(seen) == want.shape[0] == len(cfg["layers"])
    for run, (got, ref) in enumerate(zip(seen, want)):
        if dtype == "float32":
            assert float((got.cpu() - ref).abs().max()) < 1e-4, run
        else:       # a row whose router flipped may be off; most rows are not
            gap = (got.cpu() - ref).abs().amax(-1)
            assert float(gap.median()) < 0.03 * float(ref.abs().max()), run


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("case", ["A", "B", "C", "D", "E"])
def test_prompt_then_single_tokens_over_page_and_window_borders(case, dtype, tmp_path_factory):
    model = engine(case, dtype, tmp_path_factory)
    cfg = CONFIGS[case][0]
    tokens = plain.random_prompts(cfg, [150], 4)[0]
    want = expected(case, tokens)
    cache = model.make_cache(max_tokens=192, max_seqs=1)
    slot = cache.alloc()
    rows = [model.step(cache, [slot], [tokens[:50]], "all")]
    rows += [model.step(cache, [slot], [[t]], "last") for t in tokens[50:]]         # past 64, 70, 100, 128
    close(torch.cat(rows), want, dtype, f"{case} decoded", flips=routed(cfg))
    cache.free(slot)
    slot = cache.alloc()                                                            # the same slot and pages again
    rows = [model.step(cache, [slot], [[t]], "last") for t in tokens[:80]]          # from the very first token
    close(torch.cat(rows), want[:80], dtype, f"{case} decoded from the first token", flips=routed(cfg))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("case", ["A", "B", "C", "D", "E"])
def test_portions_of_several_sizes_down_to_two_tokens(case, dtype, tmp_path_factory):
    model = engine(case, dtype, tmp_path_factory)
    cfg = CONFIGS[case][0]
    tokens = plain.random_prompts(cfg, [200], 5)[0]
    want = expected(case, tokens)
    for sizes in ([2] * 40 + [120], [63, 2, 64, 1, 70], [7, 129, 64], [199, 1], [1, 2, 1, 196]):
        cache = model.make_cache(max_tokens=256, max_seqs=1)
        slot, at, rows = cache.alloc(), 0, []
        for size in sizes:
            rows.append(model.step(cache, [slot], [tokens[at:at + size]], "all"))
            at += size
        close(torch.cat(rows), want, dtype, f"{case} portions {sizes[:4]}", flips=routed(cfg))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("case", ["A", "B", "C", "D", "E"])
def test_unequal_batches_on_slots_and_pages_used_again(case, dtype, tmp_path_factory):
    model = engine(case, dtype, tmp_path_factory)
    cfg = CONFIGS[case][0]
    requests = plain.random_prompts(cfg, [90, 1, 33, 70, 5, 129], 8)
    cache = model.make_cache(max_tokens=448, max_seqs=3)
    got = {r: [] for r in range(len(requests))}
    for batch in ([0, 1, 2], [3, 4, 5]):          # the second batch takes the slots and pages the first gave back
        slots = {r: cache.alloc() for r in batch}
        cut = {r: max(1, len(requests[r]) - 4 - 2 * (r % 3)) for r in batch}
        logits = model.step(cache, [slots[r] for r in batch], [requests[r][:cut[r]] for r in batch], "all")
        at = 0
        for r in batch:
            got[r].append(logits[at:at + cut[r]])
            at += cut[r]
        live = list(batch)
        while live:
            for r in [r for r in live if cut[r] == len(requests[r])]:
                cache.free(slots.pop(r))
                live.remove(r)
            if not live:
                break
            logits = model.step(cache, [slots[r] for r in live], [[requests[r][cut[r]]] for r in live], "last")
            for i, r in enumerate(live):
                got[r].append(logits[i:i + 1])
                cut[r] += 1
        cache.check()
    for r, tokens in enumerate(requests):
        if dtype == "float32":
            close(torch.cat(got[r]), expected(case, tokens), dtype, f"{case} batched request {r}")
    close(torch.cat([row for r in range(len(requests)) for row in got[r]]),
          torch.cat([expected(case, tokens) for tokens in requests]), dtype, f"{case} batched requests", flips=routed(cfg))


@pytest.mark.parametrize("dtype", DTYPES)
def test_batch_rows_do_not_depend_on_their_neighbours(dtype, tmp_path_factory):
    model = engine("C", dtype, tmp_path_factory)
    requests = plain.random_prompts(plain.TINY_C, [77, 12, 140], 6)
    cache = model.make_cache(max_tokens=512, max_seqs=4)
    alone = []
    for tokens in requests:
        slot = cache.alloc()
        alone.append(model.step(cache, [slot], [tokens], "all"))
        cache.free(slot)
    slots = [cache.alloc() for _ in requests]
    together = model.step(cache, slots, requests, "all")
    gap = (together - torch.cat(alone)).abs()
    if dtype == "float32":
        assert float(gap.max()) < 1e-5
    else:       # tiles of other sizes round otherwise; a router's close call may then flip a row
        assert float(gap.amax(-1).median()) < 5e-2


@pytest.mark.parametrize("dtype", DTYPES)
def test_sharp_attention_finds_far_keys_in_prompts_and_in_decoding(dtype, tmp_path_factory):
    """Sharpened queries make both softmaxes pick single keys: anywhere in a window of 200 or among the 40 kept first
    positions in the grouped attention, anywhere in a window of 300 in the latent layer, so a key that is lost, read
    from the wrong page or dropped one position early moves the logits.  float32 is held to the plain
    implementation; bfloat16 (whose rounded scores such a scale magnifies) to its own whole-prompt run, which the
    decoded run must repeat from the cache."""
    model = engine("sharp", dtype, tmp_path_factory)
    tokens = plain.random_prompts(plain.SHARP, [700], 9)[0]
    cache = model.make_cache(max_tokens=1536, max_seqs=2, max_step_tokens=700)
    whole = cache.alloc()
    whole_logits = model.step(cache, [whole], [tokens], "all")
    want = expected("sharp", tokens) if dtype == "float32" else whole_logits
    if dtype == "float32":
        close(whole_logits, want, dtype, "sharp whole", atol=3e-4)      # the effects looked for below are above 2e-2
    decoded = cache.alloc()
    rows = [model.step(cache, [decoded], [tokens[:500]], "all")]
    rows += [model.step(cache, [decoded], [[t]], "last") for t in tokens[500:]]
    close(torch.cat(rows), want, dtype, "sharp decoded", atol=3e-4)
    if dtype == "float32":
        weights = weights_of("sharp")

        def changed(path, value, since):
            cfg = copy.deepcopy(plain.SHARP)
            node = cfg["layers"]
            for key in path[:-1]:
                node = node[key]
            node[path[-1]] = value
            return float((plain.forward(cfg, weights, tokens).float()[since:] - want[since:]).abs().max())
        # the plain logits really depend on the exact size of each window and on the number of kept positions
        assert changed((0, "mixer", "left", "mask", "size"), 199, 250) > 0.02
        assert changed((0, "mixer", "left", "mask", "keep_first"), 39, 250) > 0.02
        assert changed((0, "mixer", "left", "mask", "keep_first"), 41, 250) > 0.02
        assert changed((1, "mixer", "mask", "size"), 299, 300) > 0.02
        # ... and on the state that the recurrent mixer carries from the first tokens on
        later = plain.forward(plain.SHARP, weights, tokens[600:]).float()
        assert float((later[-50:] - want[-50:]).abs().max()) > 0.02


@pytest.mark.parametrize("dtype", DTYPES)
def test_long_prompts_are_cut_and_go_round_the_ring(dtype, tmp_path_factory):
    """A prompt of 700 tokens on a cache whose passes take 256 tokens of a sequence: three portions, the third one
    written over the ring's oldest pages while the pinned first pages stay, beside a short request in the same step."""
    model = engine("C", dtype, tmp_path_factory)
    long, short = plain.random_prompts(plain.TINY_C, [700, 40], 12)
    cache = model.make_cache(max_tokens=1024, max_seqs=2)
    assert cache.max_step_tokens == 256
    assert any(group.pinned_pages == 2 and (group.pinned_pages + group.ring_len) * 64 < 700 for group in cache.kv_groups)
    slots = [cache.alloc(), cache.alloc()]
    got = model.step(cache, slots, [long, short], "all")
    close(got[:700], expected("C", long), dtype, "long prompt in portions", flips=True)
    close(got[700:], expected("C", short), dtype, "short prompt beside it", flips=True)
    more = plain.random_prompts(plain.TINY_C, [30], 13)[0]
    rows = [model.step(cache, slots[:1], [[t]], "last") for t in more]
    close(torch.cat(rows), expected("C", long + more)[700:], dtype, "single tokens after the long prompt", flips=True)


@pytest.mark.parametrize("case", ["B", "C"])
def test_long_decoding_wraps_the_ring_behind_the_pinned_pages(case, tmp_path_factory):
    """Windows of tens of positions keep a ring of a few pages per sequence, behind one or two pages of kept first
    positions; 700 single-token steps go round it many times."""
    model = engine(case, "float32", tmp_path_factory)
    cfg = CONFIGS[case][0]
    tokens = plain.random_prompts(cfg, [720], 11)[0]
    want = expected(case, tokens)
    cache = model.make_cache(max_tokens=768, max_seqs=1, max_step_tokens=16)
    slot = cache.alloc()
    rows = [model.step(cache, [slot], [tokens[:20]], "all")]
    rows += [model.step(cache, [slot], [[t]], "last") for t in tokens[20:]]
    close(torch.cat(rows), want, "float32", "long decoding", atol=2e-4)
    assert any(group.pinned_pages > 0 and 720 > (group.pinned_pages + group.ring_len) * 64 for group in cache.kv_groups)


def test_decode_steps_are_captured_as_graphs(tmp_path_factory):
    assert engine("A", "bfloat16", tmp_path_factory).decoder.graph_safe


@pytest.mark.parametrize("dtype", DTYPES)
def test_greedy_generation_through_the_entry_point(dtype, tmp_path_factory):
    for case in ("A", "C"):
        model = engine(case, dtype, tmp_path_factory)
        cfg = CONFIGS[case][0]
        prompts = plain.random_prompts(cfg, [9, 30, 3], 10)
        weights = weights_of(case)
        for use_graphs in (False, True):              # the step function, then the captured decode steps
            result = model.generate(prompts, max_new_tokens=6, use_graphs=use_graphs)
            for prompt, produced in zip(prompts, result.generated_ids):
                assert len(produced) == 6
                ids = list(prompt)
                for token in produced:
                    logits = plain.forward(cfg, weights, ids)[-1]
                    slack = 1e-4 if dtype == "float32" else 0.05 * float(logits.abs().max())
                    assert float(logits.max() - logits[token]) < slack, "the generated token is not the plain argmax"
                    ids.append(token)


def test_command_line_writes_a_random_model_and_generates_from_it(tmp_path):
    cfg = plain.TINY_B
    (tmp_path / "config.json").write_text(json.dumps(cfg))
    root = Path(__file__).resolve().parent.parent
    run = lambda *a: subprocess.run([sys.executable, "-m", "ondeviceinfer_b200", *a], cwd=root, text=True,
                                    capture_output=True, timeout=600)
    made = run("random-model", "--config", str(tmp_path / "config.json"), "--seed", "3", "--out", str(tmp_path / "model"))
    assert made.returncode == 0, made.stderr
    done = run("generate", "--model", str(tmp_path / "model"), "--prompt-ids", "5,9,2,40,7", "--dtype", "float32",
               "--max-new-tokens", "4", "--warmup-runs", "0", "--repeats", "1", "--output", str(tmp_path / "report.json"))
    assert done.returncode == 0, done.stderr
    report = json.loads((tmp_path / "report.json").read_text())
    from ondeviceinfer_b200.weights import SafetensorsSource
    source = SafetensorsSource(tmp_path / "model")
    weights = {n: source.fetch(n) for n in source.stored()}
    ids = [5, 9, 2, 40, 7]
    for token in report["measurements"][0]["output_token_ids"]:
        logits = plain.forward(cfg, weights, ids)[-1]
        assert float(logits.max() - logits[token]) < 1e-4
        ids.append(token)
    assert len(ids) == 9


def test_bf16_model_whose_prompts_go_in_chunks(tmp_path):
    """States of 64 rows: a prompt long enough for the scan in chunks of 64 tokens, then single tokens and a portion."""
    cfg = plain._config(120, 64, [
        {"type": "parallel", "mixer": plain._pair(4, 2, 16, 32, 0.25, 30, 70, 4, 20, 64, 2, 4, 1), "mlp": plain._dense(48, 1.2)},
        {"type": "parallel", "mixer": plain._pair(2, 1, 32, 16, 0.18, 129, 1, 2, 64, 128, 1, 2, 1), "mlp": None}])
    weights = plain.random_weights(cfg, 312)
    assert ops.ssd_chunk_floats(1100, 1, 4, 20, 64, 2) > 0 and ops.ssd_chunk_floats(1100, 1, 2, 64, 128, 1) > 0
    model = odi.load_resident_model(write_model_folder(tmp_path / "model", cfg, weights), dtype="bfloat16")
    tokens = plain.random_prompts(cfg, [1150], 12)[0]
    want = plain.forward(cfg, weights, tokens).float()
    cache = model.make_cache(max_tokens=1216, max_seqs=1)
    slot = cache.alloc()
    rows = [model.step(cache, [slot], [tokens[:1100]], "all")]
    rows += [model.step(cache, [slot], [[t]], "last") for t in tokens[1100:1130]]
    rows.append(model.step(cache, [slot], [tokens[1130:]], "all"))
    close(torch.cat(rows), want, "bfloat16", "a prompt in chunks, single tokens, a portion", flips=False)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("seed", range(12))
def test_models_of_random_odd_sizes(seed, dtype, tmp_path):
    """Configurations drawn from odd sizes: a prompt, then single tokens, then a portion, on a cache that a shorter
    request used before."""
    cfg = plain.random_config(seed)
    weights = plain.random_weights(cfg, 300 + seed)
    model = odi.load_resident_model(write_model_folder(tmp_path / "model", cfg, weights), dtype=dtype)
    tokens = plain.random_prompts(cfg, [150], seed)[0]
    want = plain.forward(cfg, weights, tokens).float()
    cache = model.make_cache(max_tokens=192, max_seqs=1)
    slot = cache.alloc()
    model.step(cache, [slot], [tokens[:37]], "none")
    cache.free(slot)
    slot = cache.alloc()
    rows = [model.step(cache, [slot], [tokens[:100]], "all")]
    rows += [model.step(cache, [slot], [[t]], "last") for t in tokens[100:130]]
    rows.append(model.step(cache, [slot], [tokens[130:]], "all"))
    close(torch.cat(rows), want, dtype, f"random sizes {seed}: {json.dumps(cfg)[:300]}", flips=routed(cfg))
