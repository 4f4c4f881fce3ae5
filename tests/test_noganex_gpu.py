"""The Noganex design in the engine against its plain restatement (``plain_noganex``): each mechanism alone, whole
prompts, token-by-token decoding, portions, batches of unequal requests, slots and pages used again, far keys, page
borders, the edges of chunks, the first tokens, long decoding round the ring of a chunk's pages, layers that run the
tensors of others, sizes off every multiple, and greedy generation through ``generate`` and the command line.

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
import plain_noganex as plain
from helpers import F32_ATOL, F32_RTOL, write_model_folder
from ondeviceinfer_b200.kernels import ops
from ondeviceinfer_b200.parts.linear import gated_linear

pytestmark = pytest.mark.gpu
DTYPES = ["float32", "bfloat16"]
CONFIGS = {"A": (plain.TINY_A, 61), "B": (plain.TINY_B, 62), "C": (plain.TINY_C, 63), "D": (plain.TINY_D, 64),
           "sharp": (plain.SHARP, 65)}
SHARPEN = {"sharp": 5.0}
_MODELS, _PLAIN = {}, {}


def weights_of(case):
    return plain.random_weights(*CONFIGS[case], sharpen=SHARPEN.get(case, 1.0))


def engine(case, dtype, tmp_path_factory):
    if (case, dtype) not in _MODELS:
        folder = write_model_folder(tmp_path_factory.mktemp(f"noganex_{case}"), CONFIGS[case][0], weights_of(case))
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
    """float32: |d| <= ``atol``, or the helpers' bound plus a term for the size of the logits.  bfloat16: row error relative
    to the row's size: median at most 2e-2, nine rows in ten within 6e-2 and every row within 2e-1; where the router may
    flip (``flips``: the flipped row's state reaches the rows behind it) three rows in four within 6e-2."""
    actual, reference = actual.float().cpu(), reference.float().cpu()
    assert actual.shape == reference.shape and torch.isfinite(actual).all(), what
    if dtype == "float32":
        gap = (actual - reference).abs()
        bound = F32_ATOL + F32_RTOL * reference.abs() + 1e-5 * float(reference.abs().max()) if atol is None else torch.tensor(atol)
        assert not (gap > bound).any(), f"{what}: fp32 max |d| = {float(gap.max()):.3e} at logits up to {float(reference.abs().max()):.1f}"
        return
    error = (actual - reference).norm(dim=-1) / reference.norm(dim=-1).clamp_min(1e-6)
    ranked = error.sort().values
    high = ranked[int((0.75 if flips else 0.9) * len(ranked))] if len(ranked) >= 10 else ranked[-1]
    assert float(error.median()) <= 2e-2 and (float(high) <= 6e-2 or len(ranked) < 10) and (flips or float(ranked[-1]) <= 2e-1), \
        f"{what}: bfloat16 row errors median {float(error.median()):.3e}, high {float(high):.3e}, max {float(ranked[-1]):.3e}"


def ints(*values):
    return torch.tensor(values, dtype=torch.int32, device="cuda")


def tol(dtype):
    return dict(atol=2e-5, rtol=1e-5) if dtype == torch.float32 else dict(atol=2e-2, rtol=2e-2)


# ----------------------------------------------------------------------------- kernels against plain functions


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,width", [(1, 4), (5, 37), (9, 192), (3, 2052), (2, 9000), (4, 4096)])
def test_gated_normed_outputs_join_the_stream(dtype, rows, width):
    gen = torch.Generator().manual_seed(rows * width)
    x, y, gate = (torch.randn(rows, width, generator=gen) * s for s in (3.0, 2.0, 2.0))
    y[0] *= 1e-3            # eps decides beside the mean of squares
    w = 1 + 0.3 * torch.randn(width, generator=gen)
    for gated in (True, False):
        stream, rows_out = x.clone().cuda(), torch.empty(rows, width, dtype=dtype, device="cuda")
        ops.gated_norm_add(stream, y.cuda(), gate.cuda() if gated else None, w.cuda(), 1e-5, rows_out)
        want = x.double() + (plain.gated_normed(y.double(), gate.double(), w.double(), 1e-5) if gated
                             else plain.rms_norm(y.double(), w.double(), 1e-5))
        torch.testing.assert_close(stream.cpu().double(), want, atol=2e-5, rtol=1e-5)
        torch.testing.assert_close(rows_out.cpu().double(), want, **tol(dtype))
        alone = x.clone().cuda()
        ops.gated_norm_add(alone, y.cuda(), gate.cuda() if gated else None, w.cuda(), 1e-5)
        assert torch.equal(alone, stream)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("tokens,K,F", [(1, 64, 40), (3, 36, 50), (33, 96, 72), (200, 128, 136), (1100, 128, 200), (7, 512, 1000)])
@pytest.mark.parametrize("kind", ["gelu_tanh", "silu"])
def test_gated_products_with_biases(dtype, tokens, K, F, kind):
    """Every form of the product: few tokens, split K, the many-token kernel, sizes that the tensor-core kernels refuse."""
    gen = torch.Generator().manual_seed(tokens + K)
    x = torch.randn(tokens, K, generator=gen).to(dtype)
    w = (1.5 * torch.randn(2 * F, K, generator=gen) / math.sqrt(K)).to(dtype)
    b = 0.5 * torch.randn(2 * F, generator=gen)
    for bias in (b, None):
        got = gated_linear(x.cuda(), w.cuda(), bias=None if bias is None else bias.cuda(), kind=kind)
        z = x.double() @ w.double().T + (0 if bias is None else bias.double())
        act = plain.gelu_tanh if kind == "gelu_tanh" else plain.silu
        torch.testing.assert_close(got.cpu().double(), act(z[:, :F]) * z[:, F:], **(tol(dtype) if dtype == torch.float32 else dict(atol=4e-2, rtol=3e-2)))


def test_router_with_a_correction_and_renormalised_weights():
    gen = torch.Generator().manual_seed(5)
    for n_experts, top, scale in ((8, 1, 2.5), (5, 3, 1.0), (3, 3, 0.7), (40, 6, 1.3)):
        logits = torch.randn(33, n_experts, generator=gen) * 2
        correction = 0.4 * torch.randn(n_experts, generator=gen)
        logits[4] = -60.0                      # scores so small that the 1e-20 under the sum matters little, never NaN
        ids = torch.empty(33, top, dtype=torch.int32, device="cuda")
        weights = torch.empty(33, top, dtype=torch.float32, device="cuda")
        ops.moe_route(logits.cuda(), correction.cuda(), ids, weights, n_groups=1, keep=1, sigmoid=True, renormalise=True, scale=scale)
        chosen, want = plain.router_choice(logits.double(), correction.double(), top, scale)
        assert torch.equal(ids.cpu().long(), chosen)
        torch.testing.assert_close(weights.cpu().double(), want, atol=1e-6, rtol=1e-5)
        if top < n_experts:     # the choice really depends on the correction, and the weights do not contain it
            assert not torch.equal(plain.router_choice(logits.double(), torch.zeros(n_experts).double(), top, scale)[0], chosen)
        ops.moe_route(logits.cuda(), correction.cuda(), ids, weights, n_groups=1, keep=1, sigmoid=True)
        torch.testing.assert_close(weights.cpu().double(), torch.gather(torch.sigmoid(logits.double()), 1, chosen), atol=1e-6, rtol=1e-5)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("n,H,F,experts,top,shared", [(1, 16, 8, 3, 2, 8), (9, 40, 24, 5, 3, None), (300, 64, 32, 4, 1, 40), (70, 50, 20, 6, 6, 12)])
def test_silu_experts_as_a_part(dtype, n, H, F, experts, top, shared):
    from ondeviceinfer_b200.config.specs import RoutedExpertsSpec
    from ondeviceinfer_b200.parts import Runtime, build_part
    gen = torch.Generator().manual_seed(n)
    f = plain._moe(experts, top, F, 1.6, shared)
    cfg = plain._config(8, H, [(plain._delta(1, 1, 8, 8, 1), f, None)])
    w = {k[7:]: v for k, v in plain.random_weights(cfg, n).items() if k.startswith("l0.mlp.")}
    spec = RoutedExpertsSpec(hidden_size=H, expert_size=F, num_experts=experts, num_identity=0, top_k=top, num_groups=1, keep_groups=1,
                             limit=0.0, prefix="", shared_size=shared or 0, scoring="sigmoid", expert_form="gated_silu",
                             renormalise=True, weight_scale=1.6)
    part = build_part(spec)
    kind = getattr(torch, dtype)

    class Fetch:
        matrix = staticmethod(lambda name: w[name].to(kind).cuda())
        vector = staticmethod(lambda name: w[name].float().cuda())

    part.load(Fetch, Runtime(dtype=kind, device=torch.device("cuda")))
    x = torch.randn(n, H, generator=gen).to(kind)
    want = plain.routed_feed_forward({k: v.double() for k, v in w.items()}, "", f, x.double())
    got = part.forward(x.cuda(), None, None)
    added = torch.full((n, H), 2.0, device="cuda")
    part.forward(x.cuda(), type("Ctx", (), {"residual_sumsq": None})(), added)
    torch.testing.assert_close(added - 2.0, got, atol=1e-5, rtol=1e-5)
    gap = (got.cpu().double() - want).norm(dim=-1) / want.norm(dim=-1)
    assert float(gap.median()) < (1e-5 if dtype == "float32" else 1.5e-2)
    assert dtype != "float32" or float(gap.max()) < 1e-4


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("d,dv,nq,nkv,rot", [(16, 8, 4, 2, 16), (6, 5, 3, 1, 4), (48, 64, 2, 2, 20), (20, 12, 12, 2, 0), (160, 32, 8, 1, 64),
                                             (96, 80, 5, 5, 96)])
def test_head_preparation_mixes_the_queries(dtype, d, dv, nq, nkv, rot):
    gen = torch.Generator().manual_seed(d)
    n, eps = 5, 1e-5
    scaling = dict(factor=4.0, original=64, fast=8.0, slow=1.0)
    qkv = torch.randn(n, (nq + nkv) * d + nkv * dv, generator=gen).to(dtype)
    qw, kw = 1 + 0.3 * torch.randn(nq * d, generator=gen), 1 + 0.3 * torch.randn(nkv * d, generator=gen)
    talk = torch.eye(nq) + 0.5 * torch.randn(nq, nq, generator=gen)
    lanes, v_lanes = -(-d // 16) * 16, -(-dv // 16) * 16
    pos0 = 62                                          # over a page border
    cos = sin = None
    if rot:
        f, factor = plain.ramp_frequencies(rot, 500.0, scaling)
        cos, sin = torch.empty(n, rot // 2, device="cuda"), torch.empty(n, rot // 2, device="cuda")
        ops.rope_table(torch.tensor(f, dtype=torch.float64).float().cuda(), ints(*range(pos0, pos0 + n)), cos, sin, factor)
    x = qkv.double()
    q = plain.rms_norm(x[:, :nq * d], qw.double(), eps).view(n, nq, d)
    k = plain.rms_norm(x[:, nq * d:(nq + nkv) * d], kw.double(), eps).view(n, nkv, d)
    if rot:
        q, k = (plain.rotate_half(v, rot, 500.0, scaling, first=pos0) for v in (q, k))
    for mixed in (True, False):
        width = lanes * (nkv if mixed else 1)
        q_out = torch.full((n, nq * width), 7.0, dtype=dtype, device="cuda")
        k_pool = torch.full((2, nkv, 64, lanes), 7.0, dtype=dtype, device="cuda")
        v_pool = torch.full((2, nkv, 64, v_lanes), 7.0, dtype=dtype, device="cuda")
        ops.mixed_prep(qkv.cuda(), q_out, k_pool, v_pool, qw.cuda(), kw.cuda(), talk.cuda() if mixed else None, cos, sin,
                       ints(0, 0, 0, 0, 0), ints(*range(pos0, pos0 + n)), ints(0, 2), ints(1, 0), nq=nq, nkv=nkv, d=d, dv=dv,
                       lanes=lanes, v_lanes=v_lanes, rot_dim=rot, page_size=64, ring_pages=0, write_kv=True, eps=eps)
        if mixed:
            want = torch.einsum("hjg,tjgd->thjd", talk.double().view(nq, nkv, nq // nkv), q.view(n, nkv, nq // nkv, d))
            got = q_out.cpu().double().view(n, nq, nkv, lanes)
        else:
            want, got = q, q_out.cpu().double().view(n, nq, lanes)
        torch.testing.assert_close(got[..., :d], want, **tol(dtype))
        assert float(got[..., d:].abs().sum()) == 0
        for i in range(n):
            page, at = [1, 0][(pos0 + i) // 64], (pos0 + i) % 64
            torch.testing.assert_close(k_pool[page, :, at, :d].cpu().double(), k[i], **tol(dtype))
            assert torch.equal(v_pool[page, :, at, :dv].cpu(), qkv[i, (nq + nkv) * d:].view(nkv, dv))
            assert float(k_pool[page, :, at, d:].abs().sum()) == 0 and float(v_pool[page, :, at, dv:].abs().sum()) == 0
        assert float((k_pool[0, :, 5:] - 7.0).abs().max()) == 0      # nothing else was touched


# ----------------------------------------------------------------------------- attention inside chunks, with mixed heads


def _pools(keys, values, ring, n_extra_pages=3):
    """Pages as a cache with a ring of `ring` pages would hold them after writing positions 0..L-1 in order (0: every
    page kept).  Returns (k_pool, v_pool, page list)."""
    L, nkv, d = keys.shape
    n_pages = -(-L // 64) if ring == 0 else min(-(-L // 64), ring)
    order = torch.randperm(n_pages + n_extra_pages).tolist()[:n_pages]
    k_pool = torch.full((n_pages + n_extra_pages, nkv, 64, d), 9.0, dtype=keys.dtype)      # what nobody wrote is loud
    v_pool = torch.full((n_pages + n_extra_pages, nkv, 64, values.shape[-1]), 9.0, dtype=values.dtype)
    for pos in range(L):
        entry = pos // 64 if ring == 0 else pos // 64 % ring
        k_pool[order[entry], :, pos % 64] = keys[pos]
        v_pool[order[entry], :, pos % 64] = values[pos]
    return k_pool.cuda(), v_pool.cuda(), order


CHUNK_CASES = [  # chunk, total length, tokens of the step, ring pages, splits
    (40, 150, 150, 0, 1), (40, 150, 1, 0, 1), (40, 121, 1, 0, 3), (64, 200, 100, 0, 1), (64, 193, 1, 3, 2), (64, 192, 1, 3, 2),
    (130, 500, 60, 5, 1), (130, 391, 1, 4, 2), (1, 70, 70, 0, 1), (0, 260, 140, 0, 1), (0, 260, 1, 0, 4), (300, 299, 2, 0, 1),
    (17, 20, 20, 0, 1), (128, 384, 250, 0, 1), (100, 1000, 300, 7, 1), (200, 600, 1, 0, 3), (90, 700, 17, 4, 1)]


@pytest.mark.parametrize("kind,dtype", [("cores", torch.float32), ("cores", torch.bfloat16), ("tensor", torch.bfloat16),
                                        ("tensor memory", torch.bfloat16)])
@pytest.mark.parametrize("mixed", [True, False])
@pytest.mark.parametrize("chunk,L,T,ring,splits", CHUNK_CASES)
def test_attention_inside_chunks(kind, dtype, mixed, chunk, L, T, ring, splits):
    """Against the plain masked softmax, on pages laid out as the cache lays them out (positions that left the ring are
    overwritten).  One query head asks sharply for the first key of its chunk, one for the last key of the chunk before,
    one for its own position and one for a key inside: a key dropped or kept by mistake moves the output by the size
    of a value."""
    if kind == "tensor memory" and (splits > 1 or T == 1):
        pytest.skip("the form for prompts does not cut the keys")
    gen = torch.Generator().manual_seed(chunk * 1000 + L + T)
    nq, nkv, d, dv = {"tensor memory": (8, 4, 64, 64)}.get(kind, (6, 3, 32, 16) if chunk % 2 else (20, 2, 16, 48))
    keys = torch.randn(L, nkv, d, generator=gen)
    keys = keys / keys.norm(dim=-1, keepdim=True)
    values = torch.randn(L, nkv, dv, generator=gen)
    past, rep = L - T, nq // nkv
    q = torch.randn(T, nq, nkv, d, generator=gen) * 0.2
    for i in range(T):
        p = past + i
        first = p - p % chunk if chunk else 0
        for h, target in enumerate([first, first - 1, p, (first + p) // 2]):
            if 0 <= target <= p:
                q[i, h] += (40.0 / nkv if mixed else 40.0) * keys[target]
    q, keys, values = q.to(dtype), keys.to(dtype), values.to(dtype)
    if mixed:
        scores = torch.einsum("phjd,kjd->hpk", q.double(), keys.double())
    else:
        q = torch.stack([q[:, h, h // rep] for h in range(nq)], 1)
        scores = torch.einsum("phd,khd->hpk", q.double(), keys.double().repeat_interleave(rep, 1))

    def attended(size):
        masked = scores.masked_fill(~plain.same_chunk(L, size)[past:][None], float("-inf"))
        return torch.einsum("hpk,khd->phd", torch.softmax(masked, -1), values.double().repeat_interleave(rep, 1))

    want = attended(chunk or None)
    k_pool, v_pool, pages = _pools(keys, values, ring)
    out = torch.empty(T, nq * dv, dtype=dtype, device="cuda")
    partial = torch.empty(T * nq * splits * (dv + 2), device="cuda") if splits > 1 else None
    args = (q.reshape(T, -1).cuda(), k_pool, v_pool, out, ints(0, T), ints(past), ints(0, len(pages)), ints(*pages))
    common = dict(n_seqs=1, max_q_len=T, nq=nq, nkv=nkv, d=d, page_size=64, ring_pages=ring, chunk=chunk, scale=1.0, mixed=mixed)
    if kind == "cores":
        ops.attention_simt(*args, window=0, dv=dv, splits=splits, partial=partial, **common)
    elif kind == "tensor":
        ops.attention_mixed(*args, dv=dv, splits=splits, partial=partial, **common)
    else:
        ops.attention_tcgen05(*args, **common)
    torch.cuda.synchronize()
    ops.raise_on_kernel_fault()
    assert float((out.cpu().double().view(T, nq, dv) - want).abs().max()) < (1e-4 if dtype == torch.float32 else 4e-2)
    # the setup shows a chunk that is one off, and one that is counted from the portion's start
    if chunk > 1 and L > chunk and T > 1:
        assert float((attended(chunk + 1) - want).abs().max()) > 0.1
        assert float((attended(chunk - 1) - want).abs().max()) > 0.1


@pytest.mark.parametrize("kind", ["cores", "tensor", "tensor memory"])
@pytest.mark.parametrize("nq,nkv,d", [(8, 4, 128), (6, 3, 64), (8, 8, 128), (12, 6, 128), (16, 16, 64)])
def test_attention_of_unequal_sequences_in_one_launch(kind, nq, nkv, d):
    """Sequences of other lengths and pasts beside each other, with few and with many key heads (which fill the key ring
    several times a page, and leave room for 128 or for 64 query rows of all of them)."""
    gen = torch.Generator().manual_seed(3)
    chunk, dtype = 100, torch.bfloat16
    runs, pasts = [70, 1, 200, 33], [0, 99, 40, 300]
    seqs, qs, pools = [], [], []
    for T, past in zip(runs, pasts):
        L = T + past
        keys = (torch.randn(L, nkv, d, generator=gen) / math.sqrt(d)).to(dtype)
        values = torch.randn(L, nkv, d, generator=gen).to(dtype)
        q = (3.0 * torch.randn(T, nq, nkv, d, generator=gen)).to(dtype)
        scores = torch.einsum("phjd,kjd->hpk", q.double(), keys.double()).masked_fill(~plain.same_chunk(L, chunk)[past:][None], float("-inf"))
        seqs.append(torch.einsum("hpk,khd->phd", torch.softmax(scores, -1), values.double().repeat_interleave(nq // nkv, 1)))
        qs.append(q)
        pools.append(_pools(keys, values, 0, 0))
    starts, cu = [0], [0]
    for T, (_, _, order) in zip(runs, pools):
        starts.append(starts[-1] + len(order))
        cu.append(cu[-1] + T)
    ids = [starts[i] + page for i, (_, _, order) in enumerate(pools) for page in order]
    q = torch.cat(qs).reshape(cu[-1], -1).cuda()
    out = torch.empty(cu[-1], nq * d, dtype=dtype, device="cuda")
    args = (q, torch.cat([p[0] for p in pools]), torch.cat([p[1] for p in pools]), out, ints(*cu), ints(*pasts), ints(*starts), ints(*ids))
    common = dict(n_seqs=4, max_q_len=200, nq=nq, nkv=nkv, d=d, page_size=64, ring_pages=0, chunk=chunk, scale=1.0, mixed=True)
    if kind == "cores":
        ops.attention_simt(*args, window=0, dv=d, **common)
    elif kind == "tensor":
        ops.attention_mixed(*args, dv=d, **common)
    else:
        ops.attention_tcgen05(*args, **common)
    torch.cuda.synchronize()
    ops.raise_on_kernel_fault()
    assert float((out.cpu().double().view(-1, nq, d) - torch.cat(seqs)).abs().max()) < 4e-2


def test_widths_that_the_tensor_core_forms_refuse():
    assert ops.attention_mixed_supported(torch.bfloat16, 128, 128, 7, True)
    assert not ops.attention_mixed_supported(torch.bfloat16, 128, 128, 64, True)
    assert ops.attention_mixed_supported(torch.bfloat16, 128, 128, 64, False)
    assert [ops.attention_tcgen05_mixed_rows(128, n) for n in (1, 4, 5, 8, 9)] == [128, 128, 64, 64, 0]
    assert [ops.attention_tcgen05_mixed_rows(64, n) for n in (8, 16, 32)] == [128, 64, 0] and ops.attention_tcgen05_mixed_rows(48, 1) == 0


# ----------------------------------------------------------------------------- the delta rule


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("heads,kv_heads,d,dv,taps", [(4, 2, 32, 48, 3), (3, 1, 10, 7, 1), (6, 3, 24, 40, 4), (2, 2, 64, 33, 2), (4, 1, 128, 64, 4),
                                                      (1, 1, 130, 5, 16), (2, 1, 300, 16, 2), (2, 2, 16, 128, 5),
                                                      (10, 5, 128, 96, 3), (12, 4, 60, 130, 2), (40, 8, 120, 64, 2), (30, 30, 20, 90, 3),
                                                      (40, 4, 250, 64, 2)])
def test_delta_rule_over_cut_sequences(dtype, heads, kv_heads, d, dv, taps):
    """Three sequences cut into unequal runs (one token, fewer tokens than taps, groups of four with and without tokens
    left over, more than a staged chunk), stepped together with the state carried in slots of their own, against the
    recurrence over each whole sequence."""
    gen = torch.Generator().manual_seed(heads * d + dv)
    qk, v = kv_heads * d, heads * dv
    C = 2 * qk + v
    lengths = [70, 3, 31]
    projs = [torch.randn(L, C + v, generator=gen).to(dtype) for L in lengths]
    abs_ = [torch.randn(L, 2 * heads, generator=gen) for L in lengths]
    w = {"taps": torch.randn(C, taps, generator=gen) * 0.5, "A_log": torch.log(0.03 + torch.rand(heads, generator=gen)),
         "dt_bias": torch.randn(heads, generator=gen) * 0.5 - 1, "norm": 1 + 0.1 * torch.randn(dv, generator=gen)}
    m = {"heads": heads, "kv_heads": kv_heads, "dim": d, "vdim": dv}
    want = [plain.delta_core(m, p.double()[:, :C], ab.double()[:, heads:], ab.double()[:, :heads], p.double()[:, C:],
                             w["taps"].double(), w["A_log"].double(), w["dt_bias"].double(), w["norm"].double(), 1e-5)
            for p, ab in zip(projs, abs_)]
    dev = {k: t.float().cuda() for k, t in w.items()}
    dev["taps"] = dev["taps"].t().contiguous()
    slots = [4, 0, 2]
    state = torch.zeros(6, heads, d, dv, device="cuda")
    conv_state = torch.zeros(6, taps - 1, C, device="cuda") if taps > 1 else None
    state[1].fill_(7.0)          # a slot of somebody else: must stay as it is
    cuts = [[1, 1, 41, 6, 21], [1, 1, 1], [22, 1, 3, 4, 1]]
    got, at = [[] for _ in lengths], [0, 0, 0]
    for step in range(5):
        live = [s for s in range(3) if step < len(cuts[s])]
        take = lambda rows: [rows[s][at[s]:at[s] + cuts[s][step]] for s in live]
        runs = take(projs)
        cu = [0]
        for r in runs:
            cu.append(cu[-1] + len(r))
        proj = torch.cat(runs).cuda()
        tok_seq = [i for i, r in enumerate(runs) for _ in range(len(r))]
        out = torch.empty(proj.shape[0], v, dtype=dtype, device="cuda")
        ops.head_delta(proj, torch.cat(take(abs_)).cuda(), dev["taps"], dev["A_log"], dev["dt_bias"], dev["norm"], conv_state, state,
                       out, ints(*cu), ints(*tok_seq), ints(*[slots[s] for s in live]), n_seqs=len(live),
                       max_q_len=max(len(r) for r in runs), heads=heads, kv_heads=kv_heads, d=d, dv=dv, eps=1e-5, unit_eps=1e-6)
        for i, s in enumerate(live):
            got[s].append(out[cu[i]:cu[i + 1]].cpu())
            at[s] += cuts[s][step]
    assert at == lengths and float((state[1] - 7.0).abs().max()) == 0
    for s in range(3):
        torch.testing.assert_close(torch.cat(got[s]).double(), want[s], **(dict(atol=2e-4, rtol=2e-4) if dtype == torch.float32
                                                                           else dict(atol=4e-2, rtol=2e-2)))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("heads,kv_heads,d,dv,taps", [(4, 2, 64, 64, 4), (3, 3, 64, 20, 1), (2, 1, 128, 100, 3), (2, 2, 128, 128, 4),
                                                       (16, 4, 64, 52, 4), (6, 3, 128, 100, 3)])      # enough heads for the wide scan
def test_delta_rule_in_chunks_of_tokens(dtype, heads, kv_heads, d, dv, taps):
    """Runs around the chunks' edges, one of a single token among them, continued by a second step, with decays from one to
    those that wipe the state; against the recurrence in 64 bits, and no further off than four tokens at a time.  A token that is
    not a number reaches no token before it."""
    gen = torch.Generator().manual_seed(heads * d + dv)
    v = heads * dv
    C, cuts, slots = 2 * kv_heads * d + v, [[691, 16, 1, 80], [64, 97, 63, 545]], [3, 0, 4, 1]
    lengths = [a + b for a, b in zip(*cuts)]
    projs = [torch.randn(L, C + v, generator=gen).to(dtype) for L in lengths]
    abs_ = [torch.randn(L, 2 * heads, generator=gen) for L in lengths]
    abs_[0][20:22, 0] = 500.0                    # wiped inside a chunk
    abs_[1][:, 0] = -80.0                        # no decay at all
    w = {"taps": torch.randn(C, taps, generator=gen) * 0.5, "A_log": torch.log(0.03 + torch.rand(heads, generator=gen)),
         "dt_bias": torch.randn(heads, generator=gen) * 0.5 - 1, "norm": 1 + 0.1 * torch.randn(dv, generator=gen)}
    m = {"heads": heads, "kv_heads": kv_heads, "dim": d, "vdim": dv}
    want = [plain.delta_core(m, p.double()[:, :C], ab.double()[:, heads:], ab.double()[:, :heads], p.double()[:, C:],
                             w["taps"].double(), w["A_log"].double(), w["dt_bias"].double(), w["norm"].double(), 1e-5)
            for p, ab in zip(projs, abs_)]
    dev = {k: t.float().cuda() for k, t in w.items()}
    dev["taps"] = dev["taps"].t().contiguous()

    def run(in_chunks, projs=projs):
        state = torch.zeros(6, heads, d, dv, device="cuda")
        state[2].fill_(7.0)                      # a slot of somebody else: must stay as it is
        conv_state = torch.zeros(6, taps - 1, C, device="cuda") if taps > 1 else None
        got, at = [[] for _ in lengths], [0] * len(lengths)
        for lens in cuts:
            cu = [0]
            for n in lens:
                cu.append(cu[-1] + n)
            piece = lambda all_: torch.cat([x[o:o + n] for x, o, n in zip(all_, at, lens)]).cuda()
            out = torch.empty(cu[-1], v, dtype=dtype, device="cuda")
            ops.head_delta(piece(projs), piece(abs_), dev["taps"], dev["A_log"], dev["dt_bias"], dev["norm"], conv_state, state, out,
                           ints(*cu), ints(*[s for s, n in enumerate(lens) for _ in range(n)]), ints(*slots), n_seqs=len(lens),
                           max_q_len=max(lens), heads=heads, kv_heads=kv_heads, d=d, dv=dv, eps=1e-5, unit_eps=1e-6,
                           in_chunks=in_chunks)
            for s, n in enumerate(lens):
                got[s].append(out[cu[s]:cu[s + 1]].cpu().double())
                at[s] += n
        assert at == lengths and bool((state[2] == 7.0).all())
        return [torch.cat(g) for g in got], state

    off = lambda got: [float((a - b).norm() / b.norm()) for a, b in zip(got, want)]

    assert ops.head_delta_chunk_floats(sum(cuts[0]), 4, max(cuts[0]), heads, d, dv, 1) > 0
    (chunked, state), (fours, state_fours) = run(True), run(False)
    rounding = 0.0 if dtype == torch.float32 else 2.0 ** -9      # of the output; all before it is fp32 in both
    assert max(off(chunked)) < rounding + 5e-6 and max(off(fours)) < rounding + 5e-6      # sums of a hundred products of 2^-24 each
    assert sum(off(chunked)) <= (1.25 if dtype == torch.float32 else 1.01) * sum(off(fours))
    torch.testing.assert_close(state, state_fours, atol=2e-5, rtol=2e-5)
    broken = [p.clone() for p in projs]
    broken[0][100, :C] = math.nan                # in the middle of a chunk
    got = run(True, broken)[0][0]
    assert bool(torch.equal(got[:100], chunked[0][:100])) and not bool(torch.isfinite(got[100:]).any())


@pytest.mark.parametrize("d", [64, 128])
def test_chunks_of_a_run_have_the_same_bits_beside_others(d):
    """16 heads: a run by itself has a multiprocessor for each block of the scan, four runs have not."""
    gen = torch.Generator().manual_seed(d)
    heads, lens, taps = 16, [301, 64, 517, 130], 4
    C, v = 3 * heads * d, heads * d
    proj, ab = (torch.randn(sum(lens), n, generator=gen).cuda() for n in (C + v, 2 * heads))
    proj = proj.bfloat16()
    weights = (torch.randn(taps, C, generator=gen) * 0.5, torch.log(0.03 + torch.rand(heads, generator=gen)),
               torch.randn(heads, generator=gen) * 0.5 - 1, 1 + 0.1 * torch.randn(d, generator=gen))
    weights = [w.cuda() for w in weights]

    def run(first, lens):
        cu = [0]
        for n in lens:
            cu.append(cu[-1] + n)
        state, conv_state = torch.zeros(4, heads, d, d, device="cuda"), torch.zeros(4, taps - 1, C, device="cuda")
        out = torch.empty(cu[-1], v, dtype=torch.bfloat16, device="cuda")
        ops.head_delta(proj[first:first + cu[-1]], ab[first:first + cu[-1]], *weights, conv_state, state, out, ints(*cu),
                       ints(*[s for s, n in enumerate(lens) for _ in range(n)]), ints(*range(len(lens))), n_seqs=len(lens), max_q_len=max(lens),
                       heads=heads, kv_heads=heads, d=d, dv=d, eps=1e-5, unit_eps=1e-6, in_chunks=True)
        return out, state

    out, state = run(0, lens)
    at = 0
    for i, n in enumerate(lens):
        alone, alone_state = run(at, [n])
        assert torch.equal(alone, out[at:at + n]) and torch.equal(alone_state[0], state[i])
        at += n


@pytest.mark.parametrize("d", [64, 128])
def test_chunks_are_no_further_off_than_four_tokens_at_a_time(d):
    """Read-outs of runs with memories of a few to a thousand tokens, against the recurrence in 64 bits, three seeds together."""
    heads, T, off = 8, 300, {True: 0.0, False: 0.0}
    m, C = {"heads": heads, "kv_heads": heads, "dim": d, "vdim": d}, 3 * heads * d
    for seed in range(3):
        gen = torch.Generator().manual_seed(seed)
        proj, ab = torch.randn(T, C + heads * d, generator=gen), torch.randn(T, 2 * heads, generator=gen)
        taps, norm = torch.randn(C, 4, generator=gen) * 0.3, 1 + 0.1 * torch.randn(d, generator=gen)
        dt = torch.exp(math.log(1e-3) + math.log(100.0) * torch.rand(heads, generator=gen))
        a_log, bias = torch.log(1 + 15 * torch.rand(heads, generator=gen)), dt + torch.log(-torch.expm1(-dt))
        want = plain.delta_core(m, *(t.double() for t in (proj[:, :C], ab[:, heads:], ab[:, :heads], proj[:, C:], taps, a_log, bias, norm)), 1e-5)
        for in_chunks in off:
            out = torch.empty(T, heads * d, device="cuda")
            ops.head_delta(proj.cuda(), ab.cuda(), taps.t().contiguous().cuda(), a_log.cuda(), bias.cuda(), norm.cuda(),
                           torch.zeros(1, 3, C, device="cuda"), torch.zeros(1, heads, d, d, device="cuda"), out, ints(0, T), ints(*[0] * T), ints(0),
                           n_seqs=1, max_q_len=T, heads=heads, kv_heads=heads, d=d, dv=d, eps=1e-5, unit_eps=1e-6, in_chunks=in_chunks)
            off[in_chunks] += float((out.cpu().double() - want).norm() / want.norm())
    assert off[True] <= off[False]      # 0.95 of it; with products of decays rounded at every step 1.02 to 1.04


def test_delta_rule_with_decays_down_to_zero_and_no_decay_at_all():
    """Products of decays only, no quotients: a decay that underflows wipes the state, one of 1 keeps a far write."""
    heads, d, dv, L = 2, 16, 16, 90
    gen = torch.Generator().manual_seed(1)
    proj = torch.randn(L, 2 * heads * d + 2 * heads * dv, generator=gen)
    ab = torch.randn(L, 2 * heads, generator=gen)
    ab[:, 0], ab[:, 1] = -80.0, 0.0                  # head 0: softplus 0, no decay at all
    ab[40:43, 1] = 500.0                             # head 1: wiped inside a group of four
    taps, one = torch.ones(2 * heads * d + heads * dv, 1), torch.ones(dv)
    a_log = torch.zeros(heads)
    m = {"heads": heads, "kv_heads": heads, "dim": d, "vdim": dv}
    C = taps.shape[0]
    want = plain.delta_core(m, proj.double()[:, :C], ab.double()[:, heads:], ab.double()[:, :heads], proj.double()[:, C:],
                            taps.double(), a_log.double(), a_log.double(), one.double(), 1e-5)
    state = torch.zeros(1, heads, d, dv, device="cuda")
    out = torch.empty(L, heads * dv, device="cuda")
    ops.head_delta(proj.cuda(), ab.cuda(), taps.t().contiguous().cuda(), a_log.cuda(), a_log.cuda(), one.cuda(), None, state, out, ints(0, L),
                   ints(*([0] * L)), ints(0), n_seqs=1, max_q_len=L, heads=heads, kv_heads=heads, d=d, dv=dv, eps=1e-5, unit_eps=1e-6)
    assert torch.isfinite(out).all()
    torch.testing.assert_close(out.cpu().double(), want, atol=5e-4, rtol=5e-4)


# ----------------------------------------------------------------------------- whole models


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("case", ["A", "B", "C", "D"])
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
@pytest.mark.parametrize("case", ["A", "B", "C"])
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
@pytest.mark.parametrize("case", ["A", "B", "C", "D"])
def test_prompt_then_single_tokens_over_page_and_chunk_borders(case, dtype, tmp_path_factory):
    model = engine(case, dtype, tmp_path_factory)
    cfg = CONFIGS[case][0]
    tokens = plain.random_prompts(cfg, [150], 4)[0]
    want = expected(case, tokens)
    cache = model.make_cache(max_tokens=192, max_seqs=1)
    slot = cache.alloc()
    rows = [model.step(cache, [slot], [tokens[:50]], "all")]
    rows += [model.step(cache, [slot], [[t]], "last") for t in tokens[50:]]         # past 64, 80, 90, 100, 120, 128, 130
    close(torch.cat(rows), want, dtype, f"{case} decoded", flips=routed(cfg))
    cache.free(slot)
    slot = cache.alloc()                                                            # the same slot and pages again
    rows = [model.step(cache, [slot], [[t]], "last") for t in tokens[:80]]          # from the very first token
    close(torch.cat(rows), want[:80], dtype, f"{case} decoded from the first token", flips=routed(cfg))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("case", ["A", "B", "C", "D"])
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
@pytest.mark.parametrize("case", ["A", "B", "C", "D"])
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
def test_sharp_attention_finds_keys_anywhere_in_its_chunk_in_prompts_and_in_decoding(dtype, tmp_path_factory):
    """Sharpened queries make both softmaxes pick single keys anywhere in chunks of 200 and 300 positions, so a key that is
    lost, read from the wrong page or dropped one position early moves the logits.  float32 is held to the plain
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

        def changed(layer, key, value, since):
            cfg = copy.deepcopy(plain.SHARP)
            node = cfg["layers"][layer]["mixer"]
            (node["mask"] if key == "size" else node)[key] = value
            return float((plain.forward(cfg, weights, tokens).float()[since:] - want[since:]).abs().max())
        # the plain logits really depend on the exact size of each chunk, decoded positions included
        for layer, size in ((0, 200), (1, 300)):
            assert changed(layer, "size", size - 1, 500) > 0.02 and changed(layer, "size", size + 1, 500) > 0.02
        # ... on every entry of the mixing matrix
        moved = dict(weights)
        moved["l0.mix.talk"] = weights["l0.mix.talk"].clone()
        moved["l0.mix.talk"][1, 3] = 0
        assert float((plain.forward(plain.SHARP, moved, tokens).float() - want).abs().max()) > 0.02
        # ... and on the state that the recurrent mixer carries from the first tokens on
        later = plain.forward(plain.SHARP, weights, tokens[600:]).float()
        assert float((later[-50:] - want[-50:]).abs().max()) > 0.02


@pytest.mark.parametrize("dtype", DTYPES)
def test_long_prompts_are_cut_and_go_round_the_ring(dtype, tmp_path_factory):
    """A prompt of 700 tokens on a cache whose passes take 256 tokens of a sequence: three portions, written over the
    ring's oldest pages, beside a short request in the same step."""
    model = engine("C", dtype, tmp_path_factory)
    long, short = plain.random_prompts(plain.TINY_C, [700, 40], 12)
    cache = model.make_cache(max_tokens=1024, max_seqs=2)
    assert cache.max_step_tokens == 256 and any(group.ring_len * 64 < 700 for group in cache.kv_groups)
    slots = [cache.alloc(), cache.alloc()]
    got = model.step(cache, slots, [long, short], "all")
    close(got[:700], expected("C", long), dtype, "long prompt in portions", flips=True)
    close(got[700:], expected("C", short), dtype, "short prompt beside it", flips=True)
    more = plain.random_prompts(plain.TINY_C, [30], 13)[0]
    rows = [model.step(cache, slots[:1], [[t]], "last") for t in more]
    close(torch.cat(rows), expected("C", long + more)[700:], dtype, "single tokens after the long prompt", flips=True)


@pytest.mark.parametrize("case", ["B", "C"])
def test_long_decoding_wraps_the_ring(case, tmp_path_factory):
    """Chunks of tens of positions keep a ring of a few pages per sequence; 700 single-token steps go round it many times."""
    model = engine(case, "float32", tmp_path_factory)
    cfg = CONFIGS[case][0]
    tokens = plain.random_prompts(cfg, [720], 11)[0]
    cache = model.make_cache(max_tokens=768, max_seqs=1, max_step_tokens=16)
    slot = cache.alloc()
    rows = [model.step(cache, [slot], [tokens[:20]], "all")]
    rows += [model.step(cache, [slot], [[t]], "last") for t in tokens[20:]]
    close(torch.cat(rows), expected(case, tokens), "float32", "long decoding", atol=2e-4)
    assert any(720 > group.ring_len * 64 > 0 for group in cache.kv_groups)


def test_decode_steps_are_captured_as_graphs(tmp_path_factory):
    assert engine("A", "bfloat16", tmp_path_factory).decoder.graph_safe


@pytest.mark.parametrize("dtype", DTYPES)
def test_greedy_generation_through_the_entry_point(dtype, tmp_path_factory):
    for case in ("A", "C", "D"):
        model = engine(case, dtype, tmp_path_factory)
        cfg = CONFIGS[case][0]
        prompts = plain.random_prompts(cfg, [9, 60, 3], 10)
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
    """Heads of 64 and of 128: a prompt and a portion long enough for chunks of 16 tokens, single tokens between them."""
    cfg = plain._config(97, 64, [(plain._delta(2, 1, 64, 36, 4), plain._dense(48), None), (plain._delta(1, 1, 128, 20, 3), None, None)])
    weights = plain.random_weights(cfg, 313)
    assert all(ops.head_delta_chunk_floats(n, 1, n, h, d, v) > 0 for n in (240, 235) for h, d, v in ((2, 64, 36), (1, 128, 20)))
    model = odi.load_resident_model(write_model_folder(tmp_path / "model", cfg, weights), dtype="bfloat16")
    tokens = plain.random_prompts(cfg, [505], 12)[0]
    want = plain.forward(cfg, weights, tokens).float()
    cache = model.make_cache(max_tokens=512, max_seqs=1)
    slot = cache.alloc()
    rows = [model.step(cache, [slot], [tokens[:240]], "all")]
    rows += [model.step(cache, [slot], [[t]], "last") for t in tokens[240:270]]
    rows.append(model.step(cache, [slot], [tokens[270:]], "all"))
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
